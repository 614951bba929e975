// Engine core: device buffers of a lattice, groups of resident lattices with
// persistent multi-lattice launches and CUDA-graph capture, and the C ABI for
// contexts, lattices, the flow loop, measurements and diagnostics.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <new>
#include <string>
#include <type_traits>
#include <vector>

#include "lgf_engine.cuh"
#include "lgf_tiles.h"

namespace lgf {

int set_error(lgf_ctx* ctx, int code, const char* fmt, ...) {
    if (ctx) {
        char buf[512];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, sizeof buf, fmt, ap);
        va_end(ap);
        ctx->err = buf;
    }
    return code;
}

bool valid_shape(const int shape[4]) {
    if (!shape) return false;
    long long v = 1;
    for (int d = 0; d < 4; ++d) {
        if (shape[d] < 4 || (shape[d] % 2) != 0) return false;  // Lattice.cpp:42-49 (even); >= 4 for the 1x3 loops
        v *= shape[d];
    }
    return v * 4 < (1LL << 31) - 1024;  // link-thread indices are int
}

static size_t real_size(int prec) { return prec == LGF_PREC_FP64 ? sizeof(double) : sizeof(float); }

size_t footprint_bytes(const int shape[4], int precision, int meas_slots) {
    const size_t V = (size_t)shape[0] * shape[1] * shape[2] * shape[3], Vp = padded_sites(V);
    const size_t rs = real_size(precision);
    const size_t nchunk = ((size_t)shape[1] * shape[2] * shape[3] + MEAS_SITES - 1) / MEAS_SITES;
    size_t b = 3 * Vp * 4 * 18 * rs;             // link ring
    b += Vp * 4 * 8 * rs;                         // su(3) accumulator
    b += (size_t)shape[0] * nchunk * sizeof(double2) + (size_t)shape[0] * sizeof(double2);
    b += (size_t)std::max(meas_slots, 1) * (2 + 2 * (size_t)shape[0]) * sizeof(double) + 256;
    return b;
}

// Stage block size until the autotuner has run: FP64 384 threads (96 adjacent
// sites share their neighbours in L1; 7% faster per stage than 256 on 24^3x48
// and 48^4), FP32 128.  A lattice too small to fill the SMs evenly with 96-site
// tiles takes 32-site ones: the SM with the most tiles sets the time, so the
// smaller tiles are taken where they cut that SM's sites by over a tenth
// (12^4 in the staple form: 60 -> 54 us per step; 16^4, at 448 against 480
// sites, 140 either way); and 64-site ones up to one per SM (8192 sites 28.7 ->
// 26.6 us, 2 x 8^4 batched 39 -> 31).  The other stage forms have tiles of their
// own, so in a batch the sites are those that run the staple kernel together:
// 64 x 8^4, 200 steps, 113 ms with 384 threads, 121 with the 128 that one 8^4
// would take; 16 x 8^4 30.1 and 31.0; 7 x 8^4 17.8 and 14.7.
int stage_max_threads(int precision) { return precision == LGF_PREC_FP64 ? LGF_STAGE_MAXT_D : LGF_STAGE_MAXT_F; }

TileShape default_shape(int precision, long long volume) {
    const long long sms = 148;
    auto most_sites = [&](long long tile) { return ((volume + tile - 1) / tile + sms - 1) / sms * tile; };
    TileShape t;
    t.threads = 128;
    if (precision == LGF_PREC_FP64) {
        if (volume > 32 * sms && volume <= 64 * sms) t.threads = 256;
        else if (10 * most_sites(32) > 9 * most_sites(96)) t.threads = 384;
    }
    return t;
}

template <typename R> static StapleSites staple_sites_of(const std::vector<const Geom*>& members, int sms) {
    long long sites[FORMS] = {0, 0, 0, 0}, split_tiles = 0;
    for (const Geom* g : members) {
        const int form = stage_form<R>(*g);
        sites[form] += g->V;
        if (form == FORM_SPLIT) split_tiles += (g->V + SPLIT_SITES - 1) / SPLIT_SITES;
    }
    return {sites[FORM_STAPLE], sites[FORM_PARTS] + (split_tiles > sms ? sites[FORM_SPLIT] : 0)};
}
StapleSites staple_sites(int precision, const std::vector<const Geom*>& members, int sms) {
    return precision == LGF_PREC_FP64 ? staple_sites_of<double>(members, sms) : staple_sites_of<float>(members, sms);
}

static const lgf_ctx::Tuned* find_tuned(const lgf_ctx* ctx, int precision, long long volume) {
    const lgf_ctx::Tuned* best = nullptr;
    for (const auto& t : ctx->tuned)
        if (t.prec == precision && volume <= 2 * t.volume && t.volume <= 2 * volume)
            if (!best || std::llabs(t.volume - volume) < std::llabs(best->volume - volume)) best = &t;
    return best;
}

TileShape tuned_shape(const lgf_ctx* ctx, int precision, long long volume) {
    const lgf_ctx::Tuned* t = find_tuned(ctx, precision, volume);
    TileShape s = default_shape(precision, volume);
    if (!t) return s;
    if (t->stage != StageChoice::none) return t->shape;
    s.meas_budget = t->shape.meas_budget;
    s.meas_split = t->shape.meas_split;
    return s;
}

bool has_tuned(const lgf_ctx* ctx, int precision, long long volume) { return find_tuned(ctx, precision, volume) != nullptr; }
StageChoice tuned_stage(const lgf_ctx* ctx, int precision, long long volume) {
    const lgf_ctx::Tuned* t = find_tuned(ctx, precision, volume);
    return t ? t->stage : StageChoice::none;
}

void record_tuned(lgf_ctx* ctx, int precision, long long volume, const TileShape& shape, StageChoice stage) {
    for (auto& t : ctx->tuned)
        if (t.prec == precision && t.volume == volume) {
            t.shape = shape;
            t.stage = stage;
            return;
        }
    ctx->tuned.push_back({precision, volume, shape, stage});
}

void buf_free(LatticeBuf& b) {
    if (b.own_meas) cudaFree(b.meas);
    if (b.block) cudaFree(b.block);  // null: the memory belongs to the caller (a server's arena, a batch)
    b = LatticeBuf();
}

// One device allocation per lattice: each cudaMalloc or cudaFree costs ~0.15 ms
// and may stall behind other work on the device.
int buf_alloc(lgf_ctx* ctx, LatticeBuf& b, const int shape[4], int precision, int meas_slots) {
    void* block = nullptr;
    const cudaError_t e = cudaMalloc(&block, placed_bytes(shape, precision, meas_slots));
    if (e != cudaSuccess) {
        cudaGetLastError();
        b = LatticeBuf();
        return set_error(ctx, LGF_ENOMEM, "device allocation of a %dx%dx%dx%d lattice (%zu bytes) failed: %s",
                         shape[0], shape[1], shape[2], shape[3], footprint_bytes(shape, precision, meas_slots),
                         cudaGetErrorString(e));
    }
    buf_place(b, shape, precision, meas_slots, block);
    b.block = block;
    return LGF_OK;
}

// A lattice's buffers laid out inside one block of memory, each part starting
// on a 256-byte boundary (placed_bytes gives the block's size).  The link ring
// is one run: U1 (FP64) or U1..U2 (FP32) spans at least V*4*18 doubles, the
// upload/download staging area.
static inline size_t align256(size_t n) { return (n + 255) & ~size_t(255); }

size_t placed_bytes(const int shape[4], int precision, int meas_slots) {
    const size_t V = (size_t)shape[0] * shape[1] * shape[2] * shape[3], Vp = padded_sites(V);
    const size_t rs = real_size(precision);
    const size_t nchunk = ((size_t)shape[1] * shape[2] * shape[3] + MEAS_SITES - 1) / MEAS_SITES;
    return align256(3 * Vp * 4 * 18 * rs) + align256(Vp * 4 * 8 * rs) +
           align256((size_t)shape[0] * nchunk * sizeof(double2)) + align256((size_t)shape[0] * sizeof(double2)) +
           align256(2 * sizeof(int)) + align256((size_t)std::max(meas_slots, 1) * (2 + 2 * (size_t)shape[0]) * sizeof(double));
}

void buf_place(LatticeBuf& b, const int shape[4], int precision, int meas_slots, void* mem) {
    b = LatticeBuf();
    b.g = make_geom(shape);
    b.prec = precision;
    const size_t Vp = padded_sites((size_t)b.g.V), rs = real_size(precision);
    b.nchunk = (b.g.Vs + MEAS_SITES - 1) / MEAS_SITES;
    char* p = (char*)mem;
    const size_t ring = Vp * 4 * 18 * rs;
    b.U[0] = p;
    b.U[1] = p + ring;
    b.U[2] = p + 2 * ring;
    p += align256(3 * ring);
    b.A = p;
    p += align256(Vp * 4 * 8 * rs);
    b.partial = (double2*)p;
    p += align256((size_t)b.g.n[0] * b.nchunk * sizeof(double2));
    b.slice_sums = (double2*)p;
    p += align256((size_t)b.g.n[0] * sizeof(double2));
    b.slot = (int*)p;
    p += align256(2 * sizeof(int));
    b.meas_cap = std::max(meas_slots, 1);
    b.meas = (double*)p;
}

int buf_grow_meas(lgf_ctx* ctx, LatticeBuf& b, int meas_slots) {
    if (meas_slots <= b.meas_cap) return LGF_OK;
    if (!b.block) return set_error(ctx, LGF_EINVAL, "a placed lattice holds %d measurement slots", b.meas_cap);
    double* m = nullptr;
    cudaError_t e = cudaMalloc(&m, (size_t)meas_slots * (2 + 2 * (size_t)b.g.n[0]) * sizeof(double));
    if (e != cudaSuccess) {
        cudaGetLastError();
        return set_error(ctx, LGF_ENOMEM, "measurement buffer allocation failed: %s", cudaGetErrorString(e));
    }
    if (b.own_meas) cudaFree(b.meas);
    b.meas = m;
    b.own_meas = true;
    b.meas_cap = meas_slots;
    return LGF_OK;
}

int count_measurements(const lgf_flow_opts& o) {
    int n = o.measure_at_t0 ? 1 : 0;
    if (o.meas_every > 0) n += o.nsteps / o.meas_every;
    return n;
}

// The measurement lists of a subset of a group's members, assembled on the
// device from the per-member segments of the group's full measurement tile
// list (built once per change of members), so that choosing which members a
// measurement covers is one small copy and this launch, with no host wait.
//   sel = [nsel, total tiles, total slices, 0,
//          the launch segments (first tile, tiles) of the measurement kernel,
//          one pair per launch slot (read by k_measure itself),
//          then per selected member k: member, segment offset, tiles, first
//          output tile, N0, first output slice]
// Outputs: mtiles (the selected segments back to back), rtiles (member, t)
// for t < N0, counts = {tiles, slices}.  Grid
// (max(nsel, 1), any): block (k, y) copies a share of segment k.
constexpr int SEL_HEADER = 4, SEL_SEGS = 2, SEL_FIELDS = 6;  // ints; int2 segments before the launch segments; ints
__global__ void __launch_bounds__(256) k_select_measure(const int* __restrict__ sel, int fields,
                                                        const int4* __restrict__ all, int4* __restrict__ mtiles,
                                                        int2* __restrict__ rtiles, int* __restrict__ counts) {
    const int nsel = sel[0];
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        counts[0] = sel[1];
        counts[1] = sel[2];
    }
    const int k = blockIdx.x;
    if (k >= nsel) return;
    const int* f = sel + fields + SEL_FIELDS * k;
    const int member = f[0], off = f[1], n = f[2], mstart = f[3], n0 = f[4], rstart = f[5];
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < n; i += gridDim.y * blockDim.x)
        mtiles[mstart + i] = all[off + i];
    if (blockIdx.y == 0)
        for (int t = threadIdx.x; t < n0; t += blockDim.x) rtiles[rstart + t] = make_int2(member, t);
}

static inline size_t align16(size_t n) { return (n + 15) & ~size_t(15); }


// ------------------------------------------------------------------ groups
template <typename R> class Group : public GroupBase {
public:
    Group(lgf_ctx* ctx, const TileShape& shape, int max_members, long long max_tiles, bool dynamic, bool per_volume,
          int slots)
        : ctx_(ctx), shape_(shape), threads_(shape.threads), max_members_(max_members), max_tiles_(max_tiles),
          dynamic_(dynamic), per_volume_(per_volume), slots_(std::max(1, std::min(slots, max_members))),
          meas_execs_(2 * (slots_ + 1), nullptr) {}
    ~Group() override {
        cudaStreamSynchronize(ctx_->stream);  // the lists are in use until then
        drop_graphs();
        for (auto st : side_) if (st) cudaStreamDestroy(st);
        for (auto e : join_) if (e) cudaEventDestroy(e);
        if (fork_) cudaEventDestroy(fork_);
        cudaFree(d_desc_);
        cudaFree(d_tiles_);
        cudaFree(d_mtiles_);
        cudaFree(d_all_mtiles_);
        cudaFree(d_rtiles_);
        cudaFree(d_counts_);
        cudaFree(d_seg_);
        cudaFree(d_sel_);
    }

    int init() {
        LGF_CUDA_TRY(ctx_, cudaMalloc(&d_desc_, sizeof(LatDesc<R>) * max_members_));
        // a lattice takes staple tiles, or plaquette and update tiles
        const long long cap_sites = max_tiles_ * (threads_ / 4);
        tiles_cap_ = cap_sites / PLAQ_SITES + cap_sites / UPDATE_SITES + 2 * max_members_;  // the plaquette form's are the most
        LGF_CUDA_TRY(ctx_, cudaMalloc(&d_tiles_, sizeof(int2) * tiles_cap_));
        LGF_CUDA_TRY(ctx_, cudaMalloc(&d_counts_, sizeof(int) * 2));
        LGF_CUDA_TRY(ctx_, cudaMalloc(&d_seg_, sizeof(int2) * 4 * slots_));
        LGF_CUDA_TRY(ctx_, cudaMalloc(&d_sel_, sizeof(int) * sel_ints(max_members_)));
        LGF_CUDA_TRY(ctx_, cudaMemsetAsync(d_counts_, 0, sizeof(int) * 2, ctx_->stream));
        LGF_CUDA_TRY(ctx_, cudaMemsetAsync(d_sel_, 0, sizeof(int) * sel_ints(max_members_), ctx_->stream));
        if (dynamic_ && max_members_ > 1) {
            LGF_CUDA_TRY(ctx_, cudaEventCreateWithFlags(&fork_, cudaEventDisableTiming));
            for (auto& e : join_) LGF_CUDA_TRY(ctx_, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
            for (int k = 1; k >= 0; --k) LGF_CUDA_TRY(ctx_, cudaStreamCreateWithFlags(&side_[k], cudaStreamNonBlocking));
        }
        int nb = 0;
        LGF_CUDA_TRY(ctx_, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_rk3_stage<R, 1, true>, threads_, 0));
        stage_grid_max_ = std::max(1, nb) * ctx_->sm_count;
        LGF_CUDA_TRY(ctx_, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_rk3_plaquettes<R, 1>, 6 * PLAQ_SITES, 0));
        plaq_grid_max_ = std::max(1, nb) * ctx_->sm_count;
        LGF_CUDA_TRY(ctx_, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_rk3_update<R, 1>, 4 * UPDATE_SITES, 0));
        update_grid_max_ = std::max(1, nb) * ctx_->sm_count;
        // Measurement blocks: 4 tiles (loops) and 384 sites (planes) per block,
        // halved for one-warp-per-plane shapes, and smaller for lattices that
        // would not give every SM a block.
        meas_groups_ = shape_.meas_split == 2 ? LOOP_MAX_GROUPS : LOOP_MAX_GROUPS / 2;
        while (meas_groups_ > 1 && cap_sites < (long long)MEAS_SITES * meas_groups_ * ctx_->sm_count) meas_groups_ /= 2;
        unit_sites_ = shape_.meas_split == 2 ? PLANE_MAX_SITES : PLANE_MAX_SITES / 2;
        while (unit_sites_ > 96 && 3 * cap_sites < (long long)unit_sites_ * ctx_->sm_count) unit_sites_ /= 2;
        const size_t one = measure_smem_bytes<R>(), loops = loops_smem_bytes(meas_groups_), loops_most = loops_smem_bytes(LOOP_MAX_GROUPS);
        const size_t planes = planes_smem_bytes<R>(unit_sites_), planes_most = planes_smem_bytes<R>(PLANE_MAX_SITES);
        const int lt = 96 * meas_groups_;
        LGF_CUDA_TRY(ctx_, (meas_occupancy(k_measure<R, true>, MEAS_SITES * MEAS_WARPS, one, one, &nb)));
        LGF_CUDA_TRY(ctx_, (meas_occupancy(k_measure<R, false>, MEAS_SITES * MEAS_WARPS, one, one, &small_grid_max_)));
        LGF_CUDA_TRY(ctx_, (meas_occupancy(k_meas_loops<R, 0>, lt, loops, loops_most, &loops_grid_max_)));
        LGF_CUDA_TRY(ctx_, (meas_occupancy(k_meas_loops<R, 1>, lt, loops, loops_most, &nb)));
        LGF_CUDA_TRY(ctx_, (meas_occupancy(k_meas_planes<R, 0, false>, unit_sites_, planes, planes_most, &planes_grid_max_)));
        LGF_CUDA_TRY(ctx_, (meas_occupancy(k_meas_planes<R, 1, false>, unit_sites_, planes, planes_most, &nb)));
        LGF_CUDA_TRY(ctx_, (meas_occupancy(k_meas_planes<R, 0, true>, unit_sites_, planes, planes_most, &nb)));
        LGF_CUDA_TRY(ctx_, (meas_occupancy(k_meas_planes<R, 1, true>, unit_sites_, planes, planes_most, &nb)));
        if (dynamic_) {
            // members change after capture: size the measurement lists for the
            // largest resident set the tile capacity allows (x0 extents <= 256)
            mtiles_cap_ = max_tiles_ * threads_ / (4 * MEAS_SITES) + 256LL * max_members_;
            rtiles_cap_ = 256LL * max_members_;
            LGF_CUDA_TRY(ctx_, cudaMalloc(&d_mtiles_, sizeof(int4) * mtiles_cap_));
            LGF_CUDA_TRY(ctx_, cudaMalloc(&d_all_mtiles_, sizeof(int4) * mtiles_cap_));
            LGF_CUDA_TRY(ctx_, cudaMalloc(&d_rtiles_, sizeof(int2) * rtiles_cap_));
        }
        return LGF_OK;
    }

    int set_members(const std::vector<LatticeBuf*>& members) override {
        if ((int)members.size() > max_members_)
            return set_error(ctx_, LGF_EINVAL, "group holds at most %d lattices", max_members_);
        members_ = members;
        h_desc_.resize(members.size());
        std::vector<int2> tiles;
        std::vector<int4> mtiles;
        seg_off_.assign(members.size(), 0);
        seg_len_.assign(members.size(), 0);
        for (size_t i = 0; i < members.size(); ++i) {
            const LatticeBuf& b = *members[i];
            LatDesc<R>& d = h_desc_[i];
            d.g = b.g;
            d.U0 = (cplx<R>*)b.U[0];
            d.U1 = (cplx<R>*)b.U[1];
            d.U2 = (cplx<R>*)b.U[2];
            d.A = (R*)b.A;
            d.partial = b.partial;
            d.slice_sums = b.slice_sums;
            d.meas = b.meas;
            d.slot = b.slot;
            d.nchunk = b.nchunk;
            d.eps = b.eps;
            const TileShape ls = list_shape(b.g.V);
            // this member's segment of the measurement list
            seg_off_[i] = (int)mtiles.size();
            append_measure_tiles(mtiles, (int)i, b.g, ls.meas_budget, 4.0 * 18 * sizeof(R));
            seg_len_[i] = (int)mtiles.size() - seg_off_[i];
        }
        // the stage's launches, form by form (stage_form): one per run of whole
        // members, two (plaquettes, update) with the plaquette form
        std::vector<int2> segs;
        // (split lattices with more tiles than there are SMs take the staple kernel, FORM_PARTS)
        nseg_ = {0, 0, 0, 0};
        long long split_tiles = 0;
        for (auto* b : members)
            if (stage_form<R>(b->g) == FORM_SPLIT) split_tiles += (b->g.V + SPLIT_SITES - 1) / SPLIT_SITES;
        for (int form = 0; form < FORMS; ++form) {
            std::vector<int> which, len;
            for (size_t i = 0; i < members.size(); ++i) {
                int f = stage_form<R>(members[i]->g);
                if (f == FORM_SPLIT && split_tiles > ctx_->sm_count) f = FORM_PARTS;
                if (f != form) continue;
                which.push_back((int)i);
                len.push_back((members[i]->g.V + threads_ / 4 - 1) / (threads_ / 4));
            }
            if (which.empty()) continue;
            size_t m = 0;
            long long pos = 0;
            for (const int2& run : member_runs(len, slots_, 8LL * stage_grid_max_)) {
                const size_t m0 = m;
                while (m < which.size() && pos < (long long)run.x + run.y) pos += len[m++];
                for (int part = 0; part < (form == FORM_PLAQUETTE ? 2 : 1); ++part) {
                    const int first = (int)tiles.size();
                    for (size_t k = m0; k < m; ++k) {
                        const Geom& g = members[which[k]]->g;
                        if (form == FORM_PLAQUETTE) append_site_tiles(tiles, which[k], g, part ? UPDATE_SITES : PLAQ_SITES);
                        else if (form == FORM_SPLIT) append_site_tiles(tiles, which[k], g, SPLIT_SITES);
                        else append_staple_tiles(tiles, which[k], g);
                    }
                    segs.push_back(make_int2(first, (int)tiles.size() - first));
                }
                ++nseg_[form];
            }
        }
        if ((long long)tiles.size() > tiles_cap_)
            return set_error(ctx_, LGF_EINVAL, "work list of %zu tiles exceeds the group capacity %lld", tiles.size(),
                             tiles_cap_);
        const long long mt = (long long)mtiles.size();
        if (mt > mtiles_cap_) {
            if (captured()) return set_error(ctx_, LGF_EINVAL, "measurement list grew after capture");
            LGF_CUDA_TRY(ctx_, cudaStreamSynchronize(ctx_->stream));
            cudaFree(d_mtiles_);
            cudaFree(d_all_mtiles_);
            d_mtiles_ = d_all_mtiles_ = nullptr;
            LGF_CUDA_TRY(ctx_, cudaMalloc(&d_mtiles_, sizeof(int4) * std::max(mt, 1LL)));
            LGF_CUDA_TRY(ctx_, cudaMalloc(&d_all_mtiles_, sizeof(int4) * std::max(mt, 1LL)));
            mtiles_cap_ = mt;
        }
        long long rt = 0;
        for (auto* b : members) rt += b->g.n[0];
        if (rt > rtiles_cap_) {
            if (captured()) return set_error(ctx_, LGF_EINVAL, "reduction list grew after capture");
            LGF_CUDA_TRY(ctx_, cudaStreamSynchronize(ctx_->stream));
            cudaFree(d_rtiles_);
            rtiles_cap_ = std::max(rt, (long long)max_members_ * 64);
            LGF_CUDA_TRY(ctx_, cudaMalloc(&d_rtiles_, sizeof(int2) * rtiles_cap_));
        }
        ntiles_ = (int)tiles.size();
        seg_tiles_ = segs;
        // one page-locked area carries the descriptors, both tile lists and the segments
        const size_t bd = align16(sizeof(LatDesc<R>) * members.size()), bt = align16(sizeof(int2) * tiles.size()),
                     bm = align16(sizeof(int4) * mtiles.size()), bs = sizeof(int2) * segs.size();
        std::lock_guard<std::mutex> lk(ctx_->list_mu);
        char* h = nullptr;
        LGF_CUDA_TRY(ctx_, ctx_->list_stage.acquire(bd + bt + bm + bs, &h));
        std::memcpy(h, h_desc_.data(), sizeof(LatDesc<R>) * members.size());
        std::memcpy(h + bd, tiles.data(), sizeof(int2) * tiles.size());
        std::memcpy(h + bd + bt, mtiles.data(), sizeof(int4) * mtiles.size());
        std::memcpy(h + bd + bt + bm, segs.data(), bs);
        if (!members.empty())
            LGF_CUDA_TRY(ctx_, cudaMemcpyAsync(d_desc_, h, sizeof(LatDesc<R>) * members.size(), cudaMemcpyHostToDevice,
                                               ctx_->stream));
        if (ntiles_)
            LGF_CUDA_TRY(ctx_, cudaMemcpyAsync(d_tiles_, h + bd, sizeof(int2) * tiles.size(), cudaMemcpyHostToDevice,
                                               ctx_->stream));
        if (mt)
            LGF_CUDA_TRY(ctx_, cudaMemcpyAsync(d_all_mtiles_, h + bd + bt, sizeof(int4) * mtiles.size(),
                                               cudaMemcpyHostToDevice, ctx_->stream));
        if (bs) LGF_CUDA_TRY(ctx_, cudaMemcpyAsync(d_seg_, h + bd + bt + bm, bs, cudaMemcpyHostToDevice, ctx_->stream));
        LGF_CUDA_TRY(ctx_, ctx_->list_stage.release(ctx_->stream));
        return LGF_OK;
    }

    int set_eps(const std::vector<double>& eps) override {
        for (size_t i = 0; i < h_desc_.size() && i < eps.size(); ++i) h_desc_[i].eps = eps[i];
        if (h_desc_.empty()) return LGF_OK;
        std::lock_guard<std::mutex> lk(ctx_->list_mu);
        char* h = nullptr;
        LGF_CUDA_TRY(ctx_, ctx_->list_stage.acquire(sizeof(LatDesc<R>) * h_desc_.size(), &h));
        std::memcpy(h, h_desc_.data(), sizeof(LatDesc<R>) * h_desc_.size());
        LGF_CUDA_TRY(ctx_, cudaMemcpyAsync(d_desc_, h, sizeof(LatDesc<R>) * h_desc_.size(), cudaMemcpyHostToDevice,
                                           ctx_->stream));
        LGF_CUDA_TRY(ctx_, ctx_->list_stage.release(ctx_->stream));
        return LGF_OK;
    }

    // The selection table goes through a page-locked area and the lists are
    // assembled on the device (k_select_measure): no host wait.
    int set_measured(const std::vector<int>& measured) override {
        if ((int)measured.size() > max_members_) return set_error(ctx_, LGF_EINVAL, "measurement list exceeds capacity");
        for (int i : measured)
            if (i < 0 || i >= (int)members_.size()) return set_error(ctx_, LGF_EINVAL, "no member %d to measure", i);
        // small lattices (one launch) first, then the others
        std::vector<int> which(measured);
        const size_t nsmall = std::stable_partition(which.begin(), which.end(), [&](int i) { return small_measure(members_[i]->g); }) -
                              which.begin();
        std::vector<int> sel(sel_ints((int)which.size()), 0);
        std::vector<int> lens(which.size());
        PlaneMember* units[2] = {reinterpret_cast<PlaneMember*>(&sel[sel_members(0)]),
                                 reinterpret_cast<PlaneMember*>(&sel[sel_members(1)])};
        long long tm = 0, ts = 0, tr = 0, tu[2] = {0, 0};
        for (size_t k = 0; k < which.size(); ++k) {
            const int i = which[k];
            lens[k] = seg_len_[i];
            int* f = &sel[sel_fields() + SEL_FIELDS * k];
            f[0] = i;
            f[1] = seg_off_[i];
            f[2] = seg_len_[i];
            f[3] = (int)tm;
            f[4] = members_[i]->g.n[0];
            f[5] = (int)tr;
            tm += seg_len_[i];
            tr += members_[i]->g.n[0];
            if (k < nsmall) ts = tm;
            for (int round = 0; round < 2; ++round) {
                units[round][k] = {i, (int)tu[round]};
                tu[round] += plane_units(members_[i]->g, round, unit_sites_);
            }
        }
        if (tm > mtiles_cap_ || tr > rtiles_cap_ ||
            std::max(tu[0], tu[1]) > (1LL << 31) - 1024)
            return set_error(ctx_, LGF_EINVAL, "measurement list exceeds capacity");
        sel[0] = (int)which.size();
        sel[1] = (int)tm;
        sel[2] = (int)tr;
        int2* seg = reinterpret_cast<int2*>(&sel[SEL_HEADER]);
        seg[0] = make_int2(0, (int)ts);               // the small lattices' tiles
        seg[1] = make_int2((int)ts, (int)(tm - ts));  // the others'
        // the others' launch segments, in list order: runs of whole members by
        // their tiles, and the same members' plane units
        const std::vector<int2> segs = member_runs(std::vector<int>(lens.begin() + nsmall, lens.end()), slots_, 8LL * loops_grid_max_);
        size_t m = nsmall;
        long long pos = 0;
        for (size_t k = 0; k < segs.size(); ++k) {
            seg[SEL_SEGS + k] = make_int2((int)ts + segs[k].x, segs[k].y);
            const size_t m0 = m;
            while (m < which.size() && pos < (long long)segs[k].x + segs[k].y) pos += lens[m++];
            for (int round = 0; round < 2; ++round) {
                const int u0 = m0 < which.size() ? units[round][m0].start : (int)tu[round];
                const int u1 = m < which.size() ? units[round][m].start : (int)tu[round];
                seg[SEL_SEGS + (round + 1) * slots_ + k] = make_int2(u0, u1 - u0);
            }
        }
        meas_small_ = nsmall > 0;
        small_tiles_ = (int)ts;
        slice_count_ = (int)tr;
        meas_nseg_ = nsmall < which.size() ? (int)segs.size() : 0;
        {
            std::lock_guard<std::mutex> lk(ctx_->list_mu);
            char* h = nullptr;
            LGF_CUDA_TRY(ctx_, ctx_->list_stage.acquire(sizeof(int) * sel.size(), &h));
            std::memcpy(h, sel.data(), sizeof(int) * sel.size());
            LGF_CUDA_TRY(ctx_, cudaMemcpyAsync(d_sel_, h, sizeof(int) * sel.size(), cudaMemcpyHostToDevice, ctx_->stream));
            LGF_CUDA_TRY(ctx_, ctx_->list_stage.release(ctx_->stream));
        }
        k_select_measure<<<dim3(std::max<int>(1, (int)which.size()), 16), 256, 0, ctx_->stream>>>(
            d_sel_, sel_fields(), d_all_mtiles_, d_mtiles_, d_rtiles_, d_counts_);
        LGF_CUDA_TRY(ctx_, cudaGetLastError());
        return LGF_OK;
    }

    int launch_step() override { return launch_stages(); }

    // a single kernel: k = 0..2 stage k+1, k = 3 the measurement kernel alone
    // (every launch segment of it)
    int launch_one(int k) override {
        if (k < 3) {
            launch_stage(k + 1);
        } else {
            launch_measure_kernels<false>(meas_nseg_, meas_small_, MeasSites{});
        }
        LGF_CUDA_TRY(ctx_, cudaGetLastError());
        return LGF_OK;
    }

    int launch_measure() override { return launch_measurement(meas_nseg_, meas_small_); }

    // one pass over the measured members that also writes per-site outputs (single-lattice groups)
    int launch_sites(const MeasSites& out) override {
        launch_measure_kernels<true>(meas_nseg_, meas_small_, out);
        LGF_CUDA_TRY(ctx_, cudaGetLastError());
        return LGF_OK;
    }

    // drop the graphs and capture those of the current segment counts
    int capture() override {
        drop_graphs();
        int rc = capture_one(true, 0, &step_execs_[step_graph()]);
        if (rc != LGF_OK) return rc;
        return capture_one(false, meas_nseg_, &meas_execs_[meas_graph()]);
    }
    // graph launch; a graph per count of launch segments, captured on first use
    int replay_step() override {
        NvtxRange r("lgf.rk3_step");
        // a server's mixes may run through any combination of the forms' counts
        if (step_execs_.size() >= MAX_STEP_GRAPHS && !step_execs_.count(step_graph())) {
            LGF_CUDA_TRY(ctx_, cudaStreamSynchronize(ctx_->stream));  // none is running when it goes
            drop_step_graphs();
        }
        cudaGraphExec_t& g = step_execs_[step_graph()];
        if (!g) {
            int rc = capture_one(true, 0, &g);
            if (rc != LGF_OK) return rc;
        }
        LGF_CUDA_TRY(ctx_, cudaGraphLaunch(g, ctx_->stream));
        return LGF_OK;
    }
    int replay_measure() override {
        NvtxRange r("lgf.measure");
        cudaGraphExec_t& g = meas_execs_[meas_graph()];
        if (!g) {
            int rc = capture_one(false, meas_nseg_, &g);
            if (rc != LGF_OK) return rc;
        }
        LGF_CUDA_TRY(ctx_, cudaGraphLaunch(g, ctx_->stream));
        return LGF_OK;
    }
    int launches_per_step() const override { return 3 * (nseg_[FORM_STAPLE] + 2 * nseg_[FORM_PLAQUETTE] + nseg_[FORM_SPLIT] + nseg_[FORM_PARTS]); }
    int launches_per_measure() const override { return (meas_small_ ? 1 : 0) + (meas_nseg_ ? 4 * meas_nseg_ + 1 : 0) + 1; }
    int threads() const override { return threads_; }
    const TileShape& shape() const override { return shape_; }

private:
    // a measurement kernel's grid: its persistent grid, or fewer blocks when its lists are shorter
    int meas_grid(long long work, int grid_max) const {
        return dynamic_ ? grid_max : (int)std::max(1LL, std::min(work, (long long)grid_max));
    }
    // Set the kernel's shared-memory limit and find its persistent grid for this
    // group's blocks.  The limit belongs to the kernel on the device, for every
    // group and context of the process, and the last one set holds: it is the
    // most that any group's blocks take, never this group's own.
    template <typename K> cudaError_t meas_occupancy(K kernel, int threads, size_t smem, size_t most, int* grid) const {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
        int nb = 0;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, smem);
        *grid = std::max(1, nb) * ctx_->sm_count;
        return e;
    }
    // ints of a selection table for n members: header, the tiles of the small
    // and of the other lattices, the others' launch segments (loop tiles,
    // round 0 units, round 1 units), unit tables of the two rounds, member fields
    int sel_members(int round) const { return SEL_HEADER + 2 * SEL_SEGS + 6 * slots_ + 2 * max_members_ * round; }
    int sel_fields() const { return SEL_HEADER + 2 * SEL_SEGS + 6 * slots_ + 4 * max_members_; }
    size_t sel_ints(int n) const { return (size_t)sel_fields() + (size_t)SEL_FIELDS * std::max(n, 1); }
    int meas_graph() const { return 2 * meas_nseg_ + (meas_small_ ? 1 : 0); }
    bool captured() const {
        for (auto& g : step_execs_) if (g.second) return true;
        for (auto g : meas_execs_) if (g) return true;
        return false;
    }
    void drop_step_graphs() {
        for (auto& g : step_execs_) if (g.second) cudaGraphExecDestroy(g.second);
        step_execs_.clear();
    }
    void drop_graphs() {
        drop_step_graphs();
        for (auto& g : meas_execs_) if (g) { cudaGraphExecDestroy(g); g = nullptr; }
    }

    // the staple tiles of lattice i in its work order: threads_/4 consecutive
    // sites with all four link directions; per site a stage reads and writes 4
    // links and 4 su(3) accumulators
    void append_staple_tiles(std::vector<int2>& tiles, int i, const Geom& g) const {
        const TileShape ls = list_shape(g.V);
        if (!(ls.stage_order == 1 && append_stage_tiles_columns(tiles, i, g, threads_ / 4, stage_grid_max_)))
            append_stage_tiles(tiles, i, g, threads_ / 4, ls.stage_budget, 4.0 * (2 * 18 + 8) * sizeof(R));
    }
    // a stage launch's grid: persistent, or fewer blocks when its list is shorter
    int stage_grid(int j, int most) const { return dynamic_ ? most : std::max(1, std::min(seg_tiles_[j].y, most)); }
    Work stage_work(int j) const { return dynamic_ ? Work{d_seg_ + j, 0, 0} : Work{nullptr, seg_tiles_[j].x, seg_tiles_[j].y}; }
    int step_graph() const {
        int key = 0;
        for (const int n : nseg_) key = key * (slots_ + 1) + n;
        return key;
    }
    // stage S of one form's lattices: the staple form, the plaquette form's
    // pairs, the split form's (either kernel)
    template <int S> void launch_form_of(int form, cudaStream_t st) {
        int j = 0;
        for (int f = 0; f < form; ++f) j += f == FORM_PLAQUETTE ? 2 * nseg_[f] : nseg_[f];
        for (int k = 0; k < nseg_[form]; ++k) {
            if (form == FORM_PLAQUETTE) {
                k_rk3_plaquettes<R, S><<<stage_grid(j, plaq_grid_max_), 6 * PLAQ_SITES, 0, st>>>(d_desc_, d_tiles_, stage_work(j));
                ++j;
                k_rk3_update<R, S><<<stage_grid(j, update_grid_max_), 4 * UPDATE_SITES, 0, st>>>(d_desc_, d_tiles_, stage_work(j));
            } else if (form == FORM_SPLIT) {
                k_rk3_split<R, S><<<stage_grid(j, ctx_->sm_count), SPLIT_THREADS, 0, st>>>(d_desc_, d_tiles_, stage_work(j));
            } else if (form == FORM_PARTS || sizeof(R) == sizeof(float)) {  // (FP32 has no other staple form)
                k_rk3_stage<R, S, true><<<stage_grid(j, stage_grid_max_), threads_, 0, st>>>(d_desc_, d_tiles_, stage_work(j));
            } else if constexpr (sizeof(R) == sizeof(double)) {
                k_rk3_stage<R, S, false><<<stage_grid(j, stage_grid_max_), threads_, 0, st>>>(d_desc_, d_tiles_, stage_work(j));
            }
            ++j;
        }
    }
    void launch_form(int S, int form, cudaStream_t st) {
        if (S == 1) launch_form_of<1>(form, st);
        if (S == 2) launch_form_of<2>(form, st);
        if (S == 3) launch_form_of<3>(form, st);
    }
    void launch_stage(int S) {
        for (int form = 0; form < FORMS; ++form) launch_form(S, form, ctx_->stream);
    }
    // One RK3 step.  Lattices do not read one another, so the forms of a mixed
    // group run beside each other, joined at the step's end, and small
    // lattices' launches fill each other's tails.
    int launch_stages() {
        if (!dynamic_ && ntiles_ == 0) return LGF_OK;
        static const char* names[3] = {"lgf.rk3_stage1", "lgf.rk3_stage2", "lgf.rk3_stage3"};
        int forms[FORMS], n = 0;
        for (int form = 0; form < FORMS; ++form)
            if (nseg_[form]) forms[n++] = form;
        const bool beside = n > 1 && side_[0];
        if (beside) {
            LGF_CUDA_TRY(ctx_, cudaEventRecord(fork_, ctx_->stream));
            for (int k = 1; k < n; ++k) LGF_CUDA_TRY(ctx_, cudaStreamWaitEvent(side_[k - 1], fork_, 0));
        }
        for (int S = 1; S <= 3; ++S) {
            NvtxRange r(names[S - 1]);
            for (int k = 0; k < n; ++k) launch_form(S, forms[k], beside && k > 0 ? side_[k - 1] : ctx_->stream);
        }
        if (beside)
            for (int k = 1; k < n; ++k) {
                LGF_CUDA_TRY(ctx_, cudaEventRecord(join_[k - 1], side_[k - 1]));
                LGF_CUDA_TRY(ctx_, cudaStreamWaitEvent(ctx_->stream, join_[k - 1], 0));
            }
        LGF_CUDA_TRY(ctx_, cudaGetLastError());
        return LGF_OK;
    }
    int launch_measurement(int nseg, bool small) {
        NvtxRange r("lgf.measure_launch");
        launch_measure_kernels<false>(nseg, small, MeasSites{});
        return launch_reduce();
    }
    int launch_reduce() override {
        const int rg = dynamic_ ? ctx_->sm_count : std::max(1, (int)std::min<long long>(rtiles_cap_, 4 * ctx_->sm_count));
        // (the segment table stands for "read it on the device")
        const Work work = dynamic_ ? Work{d_seg_, 0, 0} : Work{nullptr, 0, slice_count_};
        k_reduce<R><<<rg, RED_THREADS, 0, ctx_->stream>>>(d_desc_, d_rtiles_, d_counts_ + 1, work);
        LGF_CUDA_TRY(ctx_, cudaGetLastError());
        return LGF_OK;
    }
    // the measurement kernels over the selection table's segments
    template <bool OUT> void launch_measure_kernels(int nseg, bool small, const MeasSites& out) {
        const int2* segs = reinterpret_cast<const int2*>(d_sel_ + SEL_HEADER);
        if (small)
            k_measure<R, OUT><<<meas_grid(mtiles_cap_, small_grid_max_), dim3(MEAS_SITES, MEAS_WARPS), measure_smem_bytes<R>(), ctx_->stream>>>(
                d_desc_, d_mtiles_, dynamic_ ? Work{segs, 0, 0} : Work{nullptr, 0, small_tiles_}, out);
        if (nseg == 0) return;
        const int2* runs = segs + SEL_SEGS;
        launch_round<0, OUT>(runs, runs + slots_, nseg, out);
        launch_round<1, OUT>(runs, runs + 2 * slots_, nseg, out);
        const int warps = SITES_THREADS / 32;
        k_meas_sites<R, OUT><<<meas_grid((mtiles_cap_ + warps - 1) / warps, 8 * ctx_->sm_count), SITES_THREADS, 0, ctx_->stream>>>(
            d_desc_, d_mtiles_, segs + 1, out);
    }
    template <int ROUND, bool OUT> void launch_round(const int2* tiles, const int2* units, int nseg, const MeasSites& out) {
        const PlaneMember* members = reinterpret_cast<const PlaneMember*>(d_sel_ + sel_members(ROUND));
        const int lg = meas_grid((mtiles_cap_ + meas_groups_ - 1) / meas_groups_, loops_grid_max_);
        const int pg = meas_grid(dynamic_ || members_.empty() ? 1 : plane_units(members_[0]->g, ROUND, unit_sites_), planes_grid_max_);
        for (int j = 0; j < nseg; ++j) {
            k_meas_loops<R, ROUND><<<lg, dim3(MEAS_SITES, 3 * meas_groups_), loops_smem_bytes(meas_groups_), ctx_->stream>>>(
                d_desc_, d_mtiles_, tiles + j);
            k_meas_planes<R, ROUND, OUT><<<pg, unit_sites_, planes_smem_bytes<R>(unit_sites_), ctx_->stream>>>(
                d_desc_, members, d_sel_, units + j, out);
        }
    }

    int capture_one(bool step, int nseg, cudaGraphExec_t* out) {
        cudaGraph_t graph = nullptr;
        LGF_CUDA_TRY(ctx_, cudaStreamBeginCapture(ctx_->stream, cudaStreamCaptureModeThreadLocal));
        int rc = step ? launch_stages() : launch_measurement(nseg, meas_small_);
        cudaError_t e = cudaStreamEndCapture(ctx_->stream, &graph);
        if (rc != LGF_OK) {
            if (graph) cudaGraphDestroy(graph);
            return rc;
        }
        if (e != cudaSuccess) return set_error(ctx_, LGF_ECUDA, "graph capture failed: %s", cudaGetErrorString(e));
        e = cudaGraphInstantiate(out, graph, 0);
        cudaGraphDestroy(graph);
        if (e != cudaSuccess) return set_error(ctx_, LGF_ECUDA, "graph instantiate failed: %s", cudaGetErrorString(e));
        return LGF_OK;
    }

    // The work order (tile order and block budgets) of one member's lists.
    // The group's shape fixes the kernels (block size, measurement split);
    // in a group of uneven volumes (per_volume_: batches, serving) each
    // member is ordered as tuned for its own volume class, else by the
    // defaults -- an order tuned on 24^3x48 (whole-slice measurement blocks)
    // costs a 48^4 member 2 to 4% in the measurement.
    TileShape list_shape(long long V) const {
        if (!per_volume_) return shape_;
        return tuned_shape(ctx_, std::is_same<R, double>::value ? LGF_PREC_FP64 : LGF_PREC_FP32MIXED, V);
    }

    lgf_ctx* ctx_;
    TileShape shape_;
    int threads_;
    int max_members_;
    long long max_tiles_;
    bool dynamic_;
    bool per_volume_;
    std::vector<LatticeBuf*> members_;
    std::vector<LatDesc<R>> h_desc_;
    std::vector<int> seg_off_, seg_len_;  // each member's segment of d_all_mtiles_
    LatDesc<R>* d_desc_ = nullptr;
    int2* d_tiles_ = nullptr;
    int4* d_mtiles_ = nullptr;      // the measured members' tiles (k_select_measure)
    int4* d_all_mtiles_ = nullptr;  // every member's measurement tiles
    int* d_sel_ = nullptr;          // selection table of the next measurement
    int2* d_rtiles_ = nullptr;
    int* d_counts_ = nullptr;  // nmtiles, nrtiles
    long long mtiles_cap_ = 0, rtiles_cap_ = 0;
    int ntiles_ = 0;
    int stage_grid_max_ = 1, small_grid_max_ = 1, loops_grid_max_ = 1, planes_grid_max_ = 1;
    int meas_groups_ = LOOP_MAX_GROUPS, unit_sites_ = PLANE_MAX_SITES;  // tiles per loops block, sites per plane unit
    int slots_;                                   // launch slots per kernel (member_runs)
    cudaStream_t side_[2] = {};                   // a mixed group's other forms (at most three forms at a time)
    cudaEvent_t fork_ = nullptr, join_[2] = {};
    std::array<int, FORMS> nseg_{};                   // stage launch segments in use, by stage form
    int meas_nseg_ = 1;                           // the measurement's
    int small_tiles_ = 0, slice_count_ = 0;       // the measured members' small tiles and x0 slices
    bool meas_small_ = false;                      // some measured lattice takes the one-launch kernel
    int2* d_seg_ = nullptr;                        // the stage's launch segments
    long long tiles_cap_ = 0;                      // capacity of d_tiles_
    int plaq_grid_max_ = 1, update_grid_max_ = 1;
    std::vector<int2> seg_tiles_;                  // tiles of each stage launch (first, count)
    static constexpr size_t MAX_STEP_GRAPHS = 64;  // as many as the counts of one form (up to 32 slots) twice over
    std::map<int, cudaGraphExec_t> step_execs_;    // by launch counts (step_graph)
    std::vector<cudaGraphExec_t> meas_execs_;      // by segment count (and small lattices)
};

GroupBase* make_group(lgf_ctx* ctx, int precision, const TileShape& shape, int max_members, long long max_tiles,
                      bool dynamic, bool per_volume, int launch_slots) {
    if (shape.threads < 128 || shape.threads % 128 || shape.threads > stage_max_threads(precision) ||
        (shape.meas_split != 1 && shape.meas_split != 2) || shape.stage_budget <= 0 || shape.meas_budget <= 0) {
        set_error(ctx, LGF_EINVAL, "invalid tile shape (threads %d, measurement split %d)", shape.threads,
                  shape.meas_split);
        return nullptr;
    }
    GroupBase* g = nullptr;
    if (precision == LGF_PREC_FP64) {
        auto* p = new (std::nothrow) Group<double>(ctx, shape, max_members, max_tiles, dynamic, per_volume, launch_slots);
        if (p && p->init() != LGF_OK) { delete p; p = nullptr; }
        g = p;
    } else {
        auto* p = new (std::nothrow) Group<float>(ctx, shape, max_members, max_tiles, dynamic, per_volume, launch_slots);
        if (p && p->init() != LGF_OK) { delete p; p = nullptr; }
        g = p;
    }
    return g;
}

// ----------------------------------------------------------- link movement
static inline int blocks_for(long long n, int t) { return (int)((n + t - 1) / t); }

// one block per 32-site layout block (the transpose kernels above)
static int launch_to_device_on(lgf_ctx* ctx, LatticeBuf& b, const double* dev_file, cudaStream_t st) {
    const int V = b.g.V;
    const int nb = blocks_for(V, LAYOUT_BLOCK);
    if (b.prec == LGF_PREC_FP64)
        k_to_device<double><<<nb, CONV_THREADS, 0, st>>>((const double2*)dev_file, (cplx<double>*)b.U[0], V);
    else
        k_to_device<float><<<nb, CONV_THREADS, 0, st>>>((const double2*)dev_file, (cplx<float>*)b.U[0], V);
    LGF_CUDA_TRY(ctx, cudaGetLastError());
    return LGF_OK;
}

int launch_to_device(lgf_ctx* ctx, LatticeBuf& b, const double* dev_file) {
    return launch_to_device_on(ctx, b, dev_file, ctx->stream);
}

int launch_to_file(lgf_ctx* ctx, const LatticeBuf& b, double* dev_file) {
    const int V = b.g.V;
    const int nb = blocks_for(V, LAYOUT_BLOCK);
    if (b.prec == LGF_PREC_FP64)
        k_to_file<double><<<nb, CONV_THREADS, 0, ctx->stream>>>((const cplx<double>*)b.U[0], (double2*)dev_file, V);
    else
        k_to_file<float><<<nb, CONV_THREADS, 0, ctx->stream>>>((const cplx<float>*)b.U[0], (double2*)dev_file, V);
    LGF_CUDA_TRY(ctx, cudaGetLastError());
    return LGF_OK;
}

int launch_generate_on(lgf_ctx* ctx, LatticeBuf& b, unsigned long long seed, double scale, cudaStream_t st) {
    const int V = b.g.V;
    if (b.prec == LGF_PREC_FP64)
        k_generate_G<double><<<blocks_for(4LL * V, 128), 128, 0, st>>>((cplx<double>*)b.U[0], V, seed, scale);
    else
        k_generate_G<float><<<blocks_for(4LL * V, 128), 128, 0, st>>>((cplx<float>*)b.U[0], V, seed, scale);
    LGF_CUDA_TRY(ctx, cudaGetLastError());
    return LGF_OK;
}

int launch_generate(lgf_ctx* ctx, LatticeBuf& b, unsigned long long seed, double scale) {
    return launch_generate_on(ctx, b, seed, scale, ctx->stream);
}

int launch_reunitarize(lgf_ctx* ctx, LatticeBuf& b) {
    const int V = b.g.V;
    if (b.prec == LGF_PREC_FP64)
        k_reunitarize<double><<<blocks_for(4LL * V, 256), 256, 0, ctx->stream>>>((cplx<double>*)b.U[0], V);
    else
        k_reunitarize<float><<<blocks_for(4LL * V, 256), 256, 0, ctx->stream>>>((cplx<float>*)b.U[0], V);
    LGF_CUDA_TRY(ctx, cudaGetLastError());
    return LGF_OK;
}

// Links cross the PCIe/C2C link as float64 file order; the reorder to the
// device layout (and the float conversion of the mixed form) runs on the GPU.
// The file-order copy is staged in the lattice's own ring: between flows the
// links live in U0 and U1 (FP64) or U1..U2 (FP32) is scratch of at least the
// file size, so an upload or download allocates no device memory.  A
// page-locked caller buffer is one DMA; pageable memory goes through the
// context's two pinned chunks, the host copy of one chunk overlapping the
// DMA of the other.
static const size_t PIN_CHUNK = 32u << 20;

static double* file_staging(const LatticeBuf& b) { return (double*)b.U[1]; }

static bool is_pinned(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost;
}

static cudaError_t ensure_pinned_chunks(lgf_ctx* ctx) {
    if (ctx->pin[0]) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < 2 && e == cudaSuccess; ++k) {
        e = cudaMallocHost(&ctx->pin[k], PIN_CHUNK);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ctx->pin_done[k], cudaEventDisableTiming);
    }
    if (e != cudaSuccess) release_pinned_chunks(ctx);
    return e;
}

void release_pinned_chunks(lgf_ctx* ctx) {
    for (int k = 0; k < 2; ++k) {
        if (ctx->pin_done[k]) cudaEventDestroy(ctx->pin_done[k]);
        if (ctx->pin[k]) cudaFreeHost(ctx->pin[k]);
        ctx->pin_done[k] = nullptr;
        ctx->pin[k] = nullptr;
    }
}

int upload_links_on(lgf_ctx* ctx, LatticeBuf& b, const double* host, cudaStream_t st) {
    const size_t bytes = (size_t)b.g.V * 4 * 18 * sizeof(double);
    char* stage = (char*)file_staging(b);
    cudaError_t e = cudaSuccess;
    if (is_pinned(host)) {
        e = cudaMemcpyAsync(stage, host, bytes, cudaMemcpyHostToDevice, st);
    } else {
        std::lock_guard<std::mutex> lk(ctx->pin_mu);
        e = ensure_pinned_chunks(ctx);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return set_error(ctx, LGF_ENOMEM, "pinned staging allocation failed: %s", cudaGetErrorString(e));
        }
        // a chunk is refilled only after the DMA that last read it (on
        // whichever stream) has finished: its event
        for (size_t off = 0, i = 0; off < bytes && e == cudaSuccess; off += PIN_CHUNK, ++i) {
            const size_t n = std::min(PIN_CHUNK, bytes - off);
            const int k = (int)(i & 1);
            e = cudaEventSynchronize(ctx->pin_done[k]);
            if (e != cudaSuccess) break;
            std::memcpy(ctx->pin[k], (const char*)host + off, n);
            e = cudaMemcpyAsync(stage + off, ctx->pin[k], n, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = cudaEventRecord(ctx->pin_done[k], st);
        }
    }
    if (e != cudaSuccess) return set_error(ctx, LGF_ECUDA, "upload failed: %s", cudaGetErrorString(e));
    return launch_to_device_on(ctx, b, (const double*)stage, st);
}

int upload_links(lgf_ctx* ctx, LatticeBuf& b, const double* host) {
    int rc = upload_links_on(ctx, b, host, ctx->stream);
    const cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (rc == LGF_OK && e != cudaSuccess) rc = set_error(ctx, LGF_ECUDA, "upload failed: %s", cudaGetErrorString(e));
    return rc;
}

// device -> host on the context's stream, complete on return: one DMA into
// page-locked memory, else through the context's two pinned chunks, the host
// copy of one overlapping the DMA of the other
int copy_out(lgf_ctx* ctx, void* host, const void* dev, size_t bytes) {
    const char* src = (const char*)dev;
    cudaError_t e = cudaSuccess;
    if (is_pinned(host)) {
        e = cudaMemcpyAsync(host, src, bytes, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    } else {
        std::lock_guard<std::mutex> lk(ctx->pin_mu);
        e = ensure_pinned_chunks(ctx);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return set_error(ctx, LGF_ENOMEM, "pinned staging allocation failed: %s", cudaGetErrorString(e));
        }
        // chunk i+1 is copied to the device-side buffer while the host drains chunk i
        const size_t nchunks = (bytes + PIN_CHUNK - 1) / PIN_CHUNK;
        auto issue = [&](size_t i) {
            const size_t off = i * PIN_CHUNK, n = std::min(PIN_CHUNK, bytes - off);
            cudaError_t r = cudaMemcpyAsync(ctx->pin[i & 1], src + off, n, cudaMemcpyDeviceToHost, ctx->stream);
            return r == cudaSuccess ? cudaEventRecord(ctx->pin_done[i & 1], ctx->stream) : r;
        };
        e = issue(0);
        for (size_t i = 0; i < nchunks && e == cudaSuccess; ++i) {
            if (i + 1 < nchunks) e = issue(i + 1);
            if (e == cudaSuccess) e = cudaEventSynchronize(ctx->pin_done[i & 1]);
            if (e != cudaSuccess) break;
            const size_t off = i * PIN_CHUNK;
            std::memcpy((char*)host + off, ctx->pin[i & 1], std::min(PIN_CHUNK, bytes - off));
        }
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    }
    if (e != cudaSuccess) return set_error(ctx, LGF_ECUDA, "copy to the host failed: %s", cudaGetErrorString(e));
    return LGF_OK;
}

int download_links(lgf_ctx* ctx, const LatticeBuf& b, double* host) {
    double* stage = file_staging(b);
    const int rc = launch_to_file(ctx, b, stage);
    return rc == LGF_OK ? copy_out(ctx, host, stage, (size_t)b.g.V * 4 * 18 * sizeof(double)) : rc;
}

}  // namespace lgf

using namespace lgf;


// =================================================================== C ABI
extern "C" {

int lgf_version(void) { return 10000; }

int lgf_ctx_create(int device, lgf_ctx** out) {
    if (!out) return LGF_EINVAL;
    *out = nullptr;
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n == 0) {
        cudaGetLastError();
        return LGF_ECUDA;
    }
    if (device < 0 || device >= n) return LGF_EINVAL;
    if (cudaSetDevice(device) != cudaSuccess) return LGF_ECUDA;
    lgf_ctx* ctx = new (std::nothrow) lgf_ctx();
    if (!ctx) return LGF_ENOMEM;
    ctx->device = device;
    if (cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaDeviceGetAttribute(&ctx->sm_count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        delete ctx;
        return LGF_ECUDA;
    }
    // place lgf_measure_noalloc's fixed scratch now, before the caller's own
    // allocations (modules load lazily otherwise)
    if (noalloc_preload(device) != LGF_OK) {
        cudaStreamDestroy(ctx->stream);
        delete ctx;
        return LGF_ECUDA;
    }
    // (without it every group pays for the chunk: no failure)
    if (cudaMalloc(&ctx->small, 256) != cudaSuccess) cudaGetLastError();
    *out = ctx;
    return LGF_OK;
}

int lgf_ctx_destroy(lgf_ctx* ctx) {
    if (!ctx) return LGF_EINVAL;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    release_pinned_chunks(ctx);
    cudaFree(ctx->small);
    cudaStreamDestroy(ctx->stream);
    delete ctx;
    return LGF_OK;
}

const char* lgf_last_error(const lgf_ctx* ctx) { return ctx ? ctx->err.c_str() : "null context"; }

size_t lgf_lattice_footprint(const int shape[4], int precision) {
    if (!valid_shape(shape) || (precision != LGF_PREC_FP64 && precision != LGF_PREC_FP32MIXED)) return 0;
    return footprint_bytes(shape, precision, 1);
}

int lgf_lattice_create(lgf_ctx* ctx, const int shape[4], int precision, lgf_lattice** out) {
    if (!ctx || !out) return LGF_EINVAL;
    *out = nullptr;
    if (!valid_shape(shape))
        return set_error(ctx, LGF_EINVAL, "lattice extents must be even and >= 4 (Lattice.cpp:42-49)");
    if (precision != LGF_PREC_FP64 && precision != LGF_PREC_FP32MIXED)
        return set_error(ctx, LGF_EINVAL, "unknown precision %d", precision);
    cudaSetDevice(ctx->device);
    lgf_lattice* lat = new (std::nothrow) lgf_lattice();
    if (!lat) return LGF_ENOMEM;
    lat->ctx = ctx;
    int rc = buf_alloc(ctx, lat->buf, shape, precision, 1);
    if (rc != LGF_OK) {
        delete lat;
        return rc;
    }
    *out = lat;
    return LGF_OK;
}

int lgf_lattice_destroy(lgf_lattice* lat) {
    if (!lat) return LGF_EINVAL;
    cudaSetDevice(lat->ctx->device);
    cudaStreamSynchronize(lat->ctx->stream);
    delete lat->group;
    buf_free(lat->buf);
    delete lat;
    return LGF_OK;
}

int lgf_upload_links(lgf_lattice* lat, const double* links) {
    if (!lat || !links) return LGF_EINVAL;
    cudaSetDevice(lat->ctx->device);
    return upload_links(lat->ctx, lat->buf, links);
}

int lgf_download_links(lgf_lattice* lat, double* links) {
    if (!lat || !links) return LGF_EINVAL;
    cudaSetDevice(lat->ctx->device);
    return download_links(lat->ctx, lat->buf, links);
}

int lgf_generate_links(lgf_lattice* lat, uint64_t seed, double scale) {
    if (!lat) return LGF_EINVAL;
    cudaSetDevice(lat->ctx->device);
    int rc = launch_generate(lat->ctx, lat->buf, seed, scale);
    if (rc != LGF_OK) return rc;
    LGF_CUDA_TRY(lat->ctx, cudaStreamSynchronize(lat->ctx->stream));
    return LGF_OK;
}

static int lattice_group(lgf_lattice* lat, GroupBase** out) {
    lgf_ctx* ctx = lat->ctx;
    const TileShape shape = tuned_shape(ctx, lat->buf.prec, lat->buf.g.V);
    if (lat->group && lat->group_shape != shape) {
        cudaStreamSynchronize(ctx->stream);
        delete lat->group;
        lat->group = nullptr;
    }
    if (!lat->group) {
        const long long ntiles = (4LL * lat->buf.g.V + shape.threads - 1) / shape.threads;
        lat->group = make_group(ctx, lat->buf.prec, shape, 1, ntiles, false);
        if (!lat->group) return ctx->err.empty() ? set_error(ctx, LGF_ENOMEM, "group creation failed") : LGF_ECUDA;
        lat->group_shape = shape;
        std::vector<LatticeBuf*> m{&lat->buf};
        int rc = lat->group->set_members(m);
        if (rc != LGF_OK) return rc;
        rc = lat->group->set_measured({0});
        if (rc != LGF_OK) return rc;
    }
    *out = lat->group;
    return LGF_OK;
}

// One measurement pass over a lattice's links with per-site (and, when asked,
// per (site, plane) F / F^) outputs, enqueued.
static int single_measure(lgf_lattice* lat, const MeasSites& out) {
    GroupBase* grp = nullptr;
    int rc = lattice_group(lat, &grp);
    return rc == LGF_OK ? grp->launch_sites(out) : rc;
}

// Where a pass leaves its site densities: the loops' scratch, dead once the
// planes are done (and free in the one-launch measurement).
static double* site_scratch(const LatticeBuf& b) { return (double*)b.U[1]; }

static int fetch_meas(lgf_ctx* ctx, const LatticeBuf& b, int nmeas, std::vector<double>& host) {
    const size_t per = 2 + 2 * (size_t)b.g.n[0];
    host.resize(per * std::max(nmeas, 1));
    if (nmeas > 0)
        LGF_CUDA_TRY(ctx, cudaMemcpyAsync(host.data(), b.meas, per * nmeas * sizeof(double), cudaMemcpyDeviceToHost,
                                          ctx->stream));
    LGF_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    return LGF_OK;
}

int lgf_flow(lgf_lattice* lat, const lgf_flow_opts* o, lgf_meas* out) {
    if (!lat || !o) return LGF_EINVAL;
    lgf_ctx* ctx = lat->ctx;
    if (o->nsteps < 0 || o->meas_every < 0 || o->reunit_every < 0)
        return set_error(ctx, LGF_EINVAL, "negative step count or interval");
    const int nmeas = count_measurements(*o);
    if (nmeas > 0) {
        if (!out || !out->t || !out->E || !out->Q)
            return set_error(ctx, LGF_EINVAL, "measurements requested but no result arrays given");
        if (out->capacity < nmeas)
            return set_error(ctx, LGF_EINVAL, "result capacity %d < %d measurements", out->capacity, nmeas);
    }
    cudaSetDevice(ctx->device);
    NvtxRange flow_range("lgf.flow");
    const double* meas_before = lat->buf.meas;
    int rc = buf_grow_meas(ctx, lat->buf, nmeas);
    if (rc != LGF_OK) return rc;
    if (lat->group && lat->buf.meas != meas_before) {
        // the measurement buffer moved: refresh the descriptor
        std::vector<LatticeBuf*> m{&lat->buf};
        rc = lat->group->set_members(m);
        if (rc != LGF_OK) return rc;
    }
    GroupBase* grp = nullptr;
    rc = lattice_group(lat, &grp);
    if (rc != LGF_OK) return rc;
    lat->buf.eps = o->eps;
    rc = grp->set_eps({o->eps});
    if (rc != LGF_OK) return rc;
    LGF_CUDA_TRY(ctx, cudaMemsetAsync(lat->buf.slot, 0, 2 * sizeof(int), ctx->stream));
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    LGF_CUDA_TRY(ctx, cudaEventCreate(&ev0));
    LGF_CUDA_TRY(ctx, cudaEventCreate(&ev1));
    struct EvGuard {
        cudaEvent_t a, b;
        ~EvGuard() { cudaEventDestroy(a); cudaEventDestroy(b); }
    } evg{ev0, ev1};
    LGF_CUDA_TRY(ctx, cudaEventRecord(ev0, ctx->stream));
    std::vector<double> tvals;
    double t = o->t0;
    if (o->measure_at_t0) {
        rc = grp->replay_measure();
        if (rc != LGF_OK) return rc;
        tvals.push_back(t);
    }
    const bool reunit = lat->buf.prec == LGF_PREC_FP32MIXED && o->reunit_every > 0;
    for (int s = 1; s <= o->nsteps; ++s) {
        rc = grp->replay_step();
        if (rc != LGF_OK) return rc;
        t += o->eps;  // GradientFlow.cpp:52
        if (reunit && s % o->reunit_every == 0) {
            rc = launch_reunitarize(ctx, lat->buf);
            if (rc != LGF_OK) return rc;
        }
        if (o->meas_every > 0 && s % o->meas_every == 0) {
            rc = grp->replay_measure();
            if (rc != LGF_OK) return rc;
            tvals.push_back(t);
        }
    }
    LGF_CUDA_TRY(ctx, cudaEventRecord(ev1, ctx->stream));
    std::vector<double> host;
    rc = fetch_meas(ctx, lat->buf, nmeas, host);
    if (rc != LGF_OK) return rc;
    float flow_ms = 0.f;
    LGF_CUDA_TRY(ctx, cudaEventElapsedTime(&flow_ms, ev0, ev1));
    lat->last_flow_s = flow_ms * 1e-3;
    if (out) {
        const int N0 = lat->buf.g.n[0];
        const size_t per = 2 + 2 * (size_t)N0;
        for (int m = 0; m < nmeas; ++m) {
            out->t[m] = tvals[m];
            out->E[m] = host[m * per + 0];
            out->Q[m] = host[m * per + 1];
            if (out->E_slice) std::memcpy(out->E_slice + (size_t)m * N0, &host[m * per + 2], N0 * sizeof(double));
            if (out->Q_slice) std::memcpy(out->Q_slice + (size_t)m * N0, &host[m * per + 2 + N0], N0 * sizeof(double));
        }
        out->count = nmeas;
    }
    return LGF_OK;
}

int lgf_measure(lgf_lattice* lat, double* E, double* Q, double* E_slice, double* Q_slice) {
    if (!lat) return LGF_EINVAL;
    lgf_flow_opts o{};
    o.eps = lat->buf.eps;
    o.nsteps = 0;
    o.measure_at_t0 = 1;
    double t, e, q;
    lgf_meas m{};
    m.capacity = 1;
    m.t = &t;
    m.E = &e;
    m.Q = &q;
    m.E_slice = E_slice;
    m.Q_slice = Q_slice;
    int rc = lgf_flow(lat, &o, &m);
    if (rc != LGF_OK) return rc;
    if (E) *E = e;
    if (Q) *Q = q;
    return LGF_OK;
}

int lgf_site_densities(lgf_lattice* lat, double* e_site, double* q_site) {
    if (!lat) return LGF_EINVAL;
    lgf_ctx* ctx = lat->ctx;
    cudaSetDevice(ctx->device);
    const size_t V = (size_t)lat->buf.g.V;
    MeasSites mo{};
    mo.e = site_scratch(lat->buf);
    mo.q = mo.e + V;
    int rc = single_measure(lat, mo);
    if (rc == LGF_OK && e_site) rc = copy_out(ctx, e_site, mo.e, V * sizeof(double));
    if (rc == LGF_OK && q_site) rc = copy_out(ctx, q_site, mo.q, V * sizeof(double));
    if (rc == LGF_OK && !e_site && !q_site) LGF_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    return rc;
}

// The same pass with the two field strengths' parts swapped (e from the
// improved F, q from the clover F), summed as a measurement is.
int lgf_measure_flowed(lgf_lattice* lat, double* E_improved, double* Q_clover) {
    if (!lat) return LGF_EINVAL;
    lgf_ctx* ctx = lat->ctx;
    cudaSetDevice(ctx->device);
    GroupBase* grp = nullptr;
    int rc = lattice_group(lat, &grp);
    if (rc != LGF_OK) return rc;
    LGF_CUDA_TRY(ctx, cudaMemsetAsync(lat->buf.slot, 0, 2 * sizeof(int), ctx->stream));
    MeasSites mo{};
    mo.swap = 1;
    rc = grp->launch_sites(mo);
    if (rc == LGF_OK) rc = grp->launch_reduce();
    std::vector<double> h;
    if (rc == LGF_OK) rc = fetch_meas(ctx, lat->buf, 1, h);
    if (rc != LGF_OK) return rc;
    if (E_improved) *E_improved = h[0];
    if (Q_clover) *Q_clover = h[1];
    return LGF_OK;
}

int lgf_last_flow_seconds(lgf_lattice* lat, double* seconds) {
    if (!lat || !seconds) return LGF_EINVAL;
    *seconds = lat->last_flow_s;
    return LGF_OK;
}

int lgf_profile_kernels(lgf_lattice* lat, double eps, int nrep, double ms[4]) {
    if (!lat || !ms || nrep < 1) return LGF_EINVAL;
    lgf_ctx* ctx = lat->ctx;
    cudaSetDevice(ctx->device);
    GroupBase* grp = nullptr;
    int rc = lattice_group(lat, &grp);
    if (rc != LGF_OK) return rc;
    lat->buf.eps = eps;
    rc = grp->set_eps({eps});
    if (rc != LGF_OK) return rc;
    LGF_CUDA_TRY(ctx, cudaMemsetAsync(lat->buf.slot, 0, 2 * sizeof(int), ctx->stream));
    std::vector<cudaEvent_t> ev(2 * 4 * nrep);
    for (auto& e : ev) LGF_CUDA_TRY(ctx, cudaEventCreate(&e));
    double acc[4] = {0, 0, 0, 0};
    cudaError_t err = cudaSuccess;
    for (int r = 0; r < nrep && rc == LGF_OK; ++r) {
        for (int k = 0; k < 4 && rc == LGF_OK; ++k) {
            cudaEventRecord(ev[(r * 4 + k) * 2], ctx->stream);
            rc = grp->launch_one(k);
            cudaEventRecord(ev[(r * 4 + k) * 2 + 1], ctx->stream);
        }
    }
    if (rc == LGF_OK) err = cudaStreamSynchronize(ctx->stream);
    if (rc == LGF_OK && err == cudaSuccess) {
        for (int r = 0; r < nrep; ++r)
            for (int k = 0; k < 4; ++k) {
                float m = 0.f;
                cudaEventElapsedTime(&m, ev[(r * 4 + k) * 2], ev[(r * 4 + k) * 2 + 1]);
                acc[k] += m;
            }
        for (int k = 0; k < 4; ++k) ms[k] = acc[k] / nrep;
    }
    for (auto& e : ev) cudaEventDestroy(e);
    if (rc != LGF_OK) return rc;
    if (err != cudaSuccess) return set_error(ctx, LGF_ECUDA, "profiling failed: %s", cudaGetErrorString(err));
    return LGF_OK;
}

int lgf_unitarity(lgf_lattice* lat, double* max_unit_err, double* max_det_err) {
    if (!lat) return LGF_EINVAL;
    lgf_ctx* ctx = lat->ctx;
    cudaSetDevice(ctx->device);
    const int V = lat->buf.g.V;
    const int nb = blocks_for(4LL * V, 256);
    double2* dp = nullptr;
    LGF_CUDA_TRY(ctx, cudaMalloc(&dp, sizeof(double2) * nb));
    if (lat->buf.prec == LGF_PREC_FP64)
        k_unitarity<double><<<nb, 256, 0, ctx->stream>>>((const cplx<double>*)lat->buf.U[0], V, dp);
    else
        k_unitarity<float><<<nb, 256, 0, ctx->stream>>>((const cplx<float>*)lat->buf.U[0], V, dp);
    std::vector<double2> h(nb);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), dp, sizeof(double2) * nb, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    cudaFree(dp);
    if (e != cudaSuccess) return set_error(ctx, LGF_ECUDA, "unitarity check failed: %s", cudaGetErrorString(e));
    double mu = 0.0, md = 0.0;
    for (const auto& v : h) {
        mu = std::max(mu, v.x);
        md = std::max(md, v.y);
    }
    if (max_unit_err) *max_unit_err = mu;
    if (max_det_err) *max_det_err = md;
    return LGF_OK;
}

int lgf_debug_gradient(lgf_lattice* lat, double* Z) {
    if (!lat || !Z) return LGF_EINVAL;
    lgf_ctx* ctx = lat->ctx;
    cudaSetDevice(ctx->device);
    const LatticeBuf& b = lat->buf;
    const size_t bytes = (size_t)b.g.V * 4 * 18 * sizeof(double);
    double2* d = nullptr;
    LGF_CUDA_TRY(ctx, cudaMalloc(&d, bytes));
    // (the plaquette form's fields go to the ring's second buffer, free between flows)
    const dim3 gp(blocks_for(b.g.V, 128), 6), gl(blocks_for(b.g.V, 128), 4);
    if (b.prec == LGF_PREC_FP64) {
        if (plaquette_stage<double>(b.g))
            k_debug_plaquettes<double><<<gp, 128, 0, ctx->stream>>>((const cplx<double>*)b.U[0], b.g, (double*)b.U[1]);
        k_debug_gradient<double><<<gl, 128, 0, ctx->stream>>>((const cplx<double>*)b.U[0], (const double*)b.U[1], b.g, d);
    } else {
        if (plaquette_stage<float>(b.g))
            k_debug_plaquettes<float><<<gp, 128, 0, ctx->stream>>>((const cplx<float>*)b.U[0], b.g, (float*)b.U[1]);
        k_debug_gradient<float><<<gl, 128, 0, ctx->stream>>>((const cplx<float>*)b.U[0], (const float*)b.U[1], b.g, d);
    }
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(Z, d, bytes, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    cudaFree(d);
    if (e != cudaSuccess) return set_error(ctx, LGF_ECUDA, "debug gradient failed: %s", cudaGetErrorString(e));
    return LGF_OK;
}

int lgf_debug_fields(lgf_lattice* lat, double* clover_F, double* improved_F) {
    if (!lat) return LGF_EINVAL;
    lgf_ctx* ctx = lat->ctx;
    cudaSetDevice(ctx->device);
    const size_t bytes = (size_t)lat->buf.g.V * 6 * 18 * sizeof(double);
    double2 *dc = nullptr, *di = nullptr;
    LGF_CUDA_TRY(ctx, cudaMalloc(&dc, bytes));
    cudaError_t e = cudaMalloc(&di, bytes);
    MeasSites mo{};
    mo.dbg_clover = dc;
    mo.dbg_improved = di;
    int rc = e == cudaSuccess ? single_measure(lat, mo)
                              : set_error(ctx, LGF_ENOMEM, "debug field buffers: %s", cudaGetErrorString(e));
    if (rc == LGF_OK) e = cudaStreamSynchronize(ctx->stream);
    if (rc == LGF_OK && e == cudaSuccess && clover_F) e = cudaMemcpy(clover_F, dc, bytes, cudaMemcpyDeviceToHost);
    if (rc == LGF_OK && e == cudaSuccess && improved_F) e = cudaMemcpy(improved_F, di, bytes, cudaMemcpyDeviceToHost);
    if (rc == LGF_OK && e != cudaSuccess) rc = set_error(ctx, LGF_ECUDA, "debug fields copy: %s", cudaGetErrorString(e));
    cudaFree(dc);
    cudaFree(di);
    return rc;
}

int lgf_exp_su3(lgf_ctx* ctx, int precision, const double* iP, double* out, long long n) {
    if (!ctx || !iP || !out || n < 0 || n > (1LL << 28)) return LGF_EINVAL;
    if (precision != LGF_PREC_FP64 && precision != LGF_PREC_FP32MIXED) return LGF_EINVAL;
    if (n == 0) return LGF_OK;
    cudaSetDevice(ctx->device);
    const size_t bytes = (size_t)n * 18 * sizeof(double);
    double2 *di = nullptr, *dout = nullptr;
    LGF_CUDA_TRY(ctx, cudaMalloc(&di, bytes));
    cudaError_t e = cudaMalloc(&dout, bytes);
    if (e == cudaSuccess) e = cudaMemcpyAsync(di, iP, bytes, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) {
        if (precision == LGF_PREC_FP64)
            k_debug_exp<double><<<blocks_for(n, 128), 128, 0, ctx->stream>>>(di, dout, (int)n);
        else
            k_debug_exp<float><<<blocks_for(n, 128), 128, 0, ctx->stream>>>(di, dout, (int)n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, dout, bytes, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    cudaFree(di);
    cudaFree(dout);
    if (e != cudaSuccess) return set_error(ctx, LGF_ECUDA, "exp failed: %s", cudaGetErrorString(e));
    return LGF_OK;
}

}  // extern "C"
