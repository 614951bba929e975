// Batched flow of many configurations of uneven volumes, and the autotuner.
//
// Jobs of one precision are packed, smallest first, into waves whose links and
// accumulators of one RK3 stage (input and output link buffers plus the su(3)
// accumulator) take at most 96 MB of the 126 MB L2.  A wave is one group:
// every RK3 stage of all its jobs is a single persistent launch over the
// wave's shared tile list, one RK3 step (its stage launches) is captured
// once as a CUDA graph and replayed, and jobs that finish early leave the
// work list (the graph reads the list and its length from device memory, so
// it is not re-captured).  Waves run one after another, so a wave's links stay
// in L2 from one stage to the next; a job too large for any wave forms a wave
// of its own (it fills the GPU alone).  Each job's arithmetic is exactly what
// lgf_flow does for it alone.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <memory>
#include <new>
#include <vector>

#include "lgf_engine.cuh"

using namespace lgf;

namespace {

struct JobRun {
    lgf_job* job;
    LatticeBuf buf;
    int nmeas = 0;
    std::vector<double> tvals;
    double t = 0.0;
};

int validate_job(lgf_ctx* ctx, const lgf_job& j) {
    if (!valid_shape(j.shape)) return set_error(ctx, LGF_EINVAL, "job lattice extents must be even and >= 4");
    if (j.precision != LGF_PREC_FP64 && j.precision != LGF_PREC_FP32MIXED)
        return set_error(ctx, LGF_EINVAL, "unknown precision %d", j.precision);
    if (j.flow.nsteps < 0 || j.flow.meas_every < 0 || j.flow.reunit_every < 0)
        return set_error(ctx, LGF_EINVAL, "negative step count or interval");
    const int nm = count_measurements(j.flow);
    if (nm > 0 && (!j.meas || !j.meas->t || !j.meas->E || !j.meas->Q || j.meas->capacity < nm))
        return set_error(ctx, LGF_EINVAL, "job result arrays missing or capacity < %d", nm);
    return LGF_OK;
}

// tile shape for waves whose largest lattice has this shape: tuned once per
// precision and volume class (stage: its stage block size too)
TileShape shape_for(lgf_ctx* ctx, int prec, const int shape[4], bool stage) {
    const long long V = 1LL * shape[0] * shape[1] * shape[2] * shape[3];
    if (has_tuned(ctx, prec, V)) return tuned_shape(ctx, prec, V);
    TileShape best = default_shape(prec, V);
    if (tune_shape(ctx, prec, shape, stage, &best) != LGF_OK) {
        ctx->err.clear();
        return default_shape(prec, V);
    }
    return best;
}

// Every job's results: runs of copies into a page-locked area of a bounded size
// (the context keeps it) with one wait each, a larger job's on its own through
// the pinned chunks, then the final links that are asked for.
constexpr size_t RESULT_AREA_BYTES = 16u << 20;

int fetch_results(lgf_ctx* ctx, std::vector<std::unique_ptr<JobRun>>& runs) {
    auto per = [](const JobRun& r) { return 2 + 2 * (size_t)r.buf.g.n[0]; };
    auto bytes = [&](const JobRun& r) { return per(r) * r.nmeas * sizeof(double); };
    auto deliver = [&](const JobRun& r, const double* v) {
        const lgf_meas* out = r.job->meas;
        const int N0 = r.buf.g.n[0];
        for (int m = 0; out && m < r.nmeas; ++m, v += per(r)) {
            out->t[m] = r.tvals[m];
            out->E[m] = v[0];
            out->Q[m] = v[1];
            if (out->E_slice) std::memcpy(out->E_slice + (size_t)m * N0, v + 2, N0 * sizeof(double));
            if (out->Q_slice) std::memcpy(out->Q_slice + (size_t)m * N0, v + 2 + N0, N0 * sizeof(double));
        }
    };
    for (size_t i = 0, j; i < runs.size(); i = j) {
        size_t total = bytes(*runs[i]);
        for (j = i + 1; j < runs.size() && total + bytes(*runs[j]) <= RESULT_AREA_BYTES; ++j) total += bytes(*runs[j]);
        if (total == 0) continue;
        if (total > RESULT_AREA_BYTES) {  // one job
            std::vector<double> h(total / sizeof(double));
            const int rc = copy_out(ctx, h.data(), runs[i]->buf.meas, total);
            if (rc != LGF_OK) return rc;
            deliver(*runs[i], h.data());
            continue;
        }
        std::lock_guard<std::mutex> lk(ctx->list_mu);
        char* h = nullptr;
        LGF_CUDA_TRY(ctx, ctx->list_stage.acquire(total, &h));
        size_t off = 0;
        for (size_t k = i; k < j; ++k) {
            const size_t n = bytes(*runs[k]);
            if (n) LGF_CUDA_TRY(ctx, cudaMemcpyAsync(h + off, runs[k]->buf.meas, n, cudaMemcpyDeviceToHost, ctx->stream));
            off += n;
        }
        LGF_CUDA_TRY(ctx, ctx->list_stage.release(ctx->stream));
        LGF_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
        off = 0;
        for (size_t k = i; k < j; ++k) {
            deliver(*runs[k], (const double*)(h + off));
            off += bytes(*runs[k]);
        }
    }
    for (const auto& r : runs) {
        if (r->job->meas) r->job->meas->count = r->nmeas;
        if (!r->job->links_out) continue;
        const int rc = download_links(ctx, r->buf, r->job->links_out);
        if (rc != LGF_OK) return rc;
    }
    return LGF_OK;
}

// Flow one wave of jobs (same precision) in lockstep on the precision's group
// (dynamic: the wave becomes its member set and the captured graphs stay
// valid); adds the kernel launches issued to *launches.
int run_wave(lgf_ctx* ctx, int prec, std::vector<JobRun*>& runs, GroupBase* grp, int* launches) {
    std::vector<LatticeBuf*> members;
    std::vector<double> eps;
    for (auto* r : runs) {
        members.push_back(&r->buf);
        eps.push_back(r->job->flow.eps);
        r->buf.eps = r->job->flow.eps;
        LGF_CUDA_TRY(ctx, cudaMemsetAsync(r->buf.slot, 0, 2 * sizeof(int), ctx->stream));
        r->t = r->job->flow.t0;
    }
    int rc = grp->set_members(members);
    if (rc != LGF_OK) return rc;
    int maxsteps = 0;
    for (auto* r : runs) maxsteps = std::max(maxsteps, r->job->flow.nsteps);

    std::vector<int> last_measured{-1};
    auto measure = [&](const std::vector<int>& which) -> int {
        if (which.empty()) return LGF_OK;
        if (which != last_measured) {
            int e = grp->set_measured(which);
            if (e != LGF_OK) return e;
            last_measured = which;
        }
        *launches += grp->launches_per_measure();
        return grp->replay_measure();
    };
    // t0 measurements
    {
        std::vector<int> which;
        for (size_t i = 0; i < runs.size(); ++i)
            if (runs[i]->job->flow.measure_at_t0) {
                which.push_back((int)i);
                runs[i]->tvals.push_back(runs[i]->t);
            }
        rc = measure(which);
        if (rc != LGF_OK) return rc;
    }
    std::vector<JobRun*> active = runs;
    for (int s = 1; s <= maxsteps; ++s) {
        // jobs whose step count is reached leave the work list
        std::vector<JobRun*> still;
        for (auto* r : active)
            if (r->job->flow.nsteps >= s) still.push_back(r);
        if (still.size() != active.size()) {
            active = still;
            members.clear();
            for (auto* r : active) members.push_back(&r->buf);
            rc = grp->set_members(members);
            if (rc != LGF_OK) return rc;
            last_measured = {-1};
        }
        if (active.empty()) break;
        rc = grp->replay_step();
        if (rc != LGF_OK) return rc;
        *launches += grp->launches_per_step();
        std::vector<int> which;
        for (size_t i = 0; i < active.size(); ++i) {
            JobRun* r = active[i];
            r->t += r->job->flow.eps;  // GradientFlow.cpp:52
            const lgf_flow_opts& o = r->job->flow;
            if (prec == LGF_PREC_FP32MIXED && o.reunit_every > 0 && s % o.reunit_every == 0) {
                rc = launch_reunitarize(ctx, r->buf);
                if (rc != LGF_OK) return rc;
                *launches += 1;
            }
            if (o.meas_every > 0 && s % o.meas_every == 0) {
                which.push_back((int)i);
                r->tvals.push_back(r->t);
            }
        }
        rc = measure(which);
        if (rc != LGF_OK) return rc;
    }
    return LGF_OK;
}

// L2-sized waves: jobs sorted by volume, packed greedily while the links and
// accumulators of a stage fit the budget; order inside a wave is the input order.
// The plaquette form's projections (half as much again) are not counted.  64
// uneven lattices, 60 steps, FP64 and FP32, ms: as it is 1089 and 638; counted
// against 96 MB 1089 and 644, 128 MB 1098 and 645, 64 MB 1105 and 646; not
// counted, 64 MB 1100 and 644, 192 MB 1104 and 642.
#ifndef LGF_BATCH_WAVE_MB
#define LGF_BATCH_WAVE_MB 96  // 0: every job of a precision in one wave
#endif
const size_t L2_WAVE_BYTES = (size_t)LGF_BATCH_WAVE_MB << 20;

std::vector<std::vector<JobRun*>> l2_waves(const std::vector<JobRun*>& jobs, int prec) {
    const size_t rs = prec == LGF_PREC_FP64 ? 8 : 4;
    auto stage_bytes = [&](const JobRun* r) { return (size_t)r->buf.g.V * 4 * (2 * 18 + 8) * rs; };
    std::vector<JobRun*> order = jobs;
    std::stable_sort(order.begin(), order.end(), [](const JobRun* a, const JobRun* b) { return a->buf.g.V < b->buf.g.V; });
    std::vector<std::vector<JobRun*>> waves;
    size_t cur = 0;
    for (JobRun* r : order) {
        const size_t b = stage_bytes(r);
        if (waves.empty() || (L2_WAVE_BYTES > 0 && cur + b > L2_WAVE_BYTES)) {
            waves.emplace_back();
            cur = 0;
        }
        waves.back().push_back(r);
        cur += b;
    }
    return waves;
}

}  // namespace

extern "C" {

int lgf_batch_run(lgf_ctx* ctx, lgf_job* jobs, int njobs, lgf_batch_stats* stats) {
    if (!ctx || (!jobs && njobs > 0) || njobs < 0) return LGF_EINVAL;
    cudaSetDevice(ctx->device);
    for (int i = 0; i < njobs; ++i) {
        int rc = validate_job(ctx, jobs[i]);
        if (rc != LGF_OK) return rc;
    }
    // one allocation holds every job (a cudaMalloc and cudaFree per buffer took
    // 18 of a 14-job ensemble's 62 ms, and each may stall for much longer)
    std::vector<size_t> at(njobs + 1, 0);
    for (int i = 0; i < njobs; ++i)
        at[i + 1] = at[i] + placed_bytes(jobs[i].shape, jobs[i].precision, count_measurements(jobs[i].flow));
    char* memory = nullptr;
    if (njobs > 0) {
        const cudaError_t e = cudaMalloc(&memory, at[njobs]);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return set_error(ctx, LGF_ENOMEM, "device allocation of %d jobs (%zu bytes) failed: %s", njobs, at[njobs], cudaGetErrorString(e));
        }
    }
    std::vector<std::unique_ptr<JobRun>> runs;
    auto cleanup = [&]() {
        cudaStreamSynchronize(ctx->stream);
        if (memory) cudaFree(memory);
    };
    double site_steps = 0.0;
    for (int i = 0; i < njobs; ++i) {
        auto r = std::make_unique<JobRun>();
        r->job = &jobs[i];
        r->nmeas = count_measurements(jobs[i].flow);
        buf_place(r->buf, jobs[i].shape, jobs[i].precision, r->nmeas, memory + at[i]);
        // (page-locked links are read by the DMA until the stream gets past it, before this call returns)
        const int rc = jobs[i].links ? upload_links_on(ctx, r->buf, jobs[i].links, ctx->stream)
                                     : launch_generate(ctx, r->buf, jobs[i].seed, jobs[i].gen_scale);
        runs.push_back(std::move(r));
        if (rc != LGF_OK) {
            cleanup();
            return rc;
        }
        site_steps += (double)runs.back()->buf.g.V * jobs[i].flow.nsteps;
    }
    // group the jobs by precision and pick each group's block size (autotuned
    // once per context, before the timed region)
    std::vector<JobRun*> groups[2];
    std::vector<std::vector<JobRun*>> waves_of[2];
    TileShape shapes[2];
    for (int prec = 0; prec < 2; ++prec) {
        int big[4] = {4, 4, 4, 4};
        long long bigV = 0;
        for (auto& r : runs)
            if (r->job->precision == prec) {
                groups[prec].push_back(r.get());
                if ((long long)r->buf.g.V > bigV) {
                    bigV = r->buf.g.V;
                    std::memcpy(big, r->job->shape, sizeof big);
                }
            }
        if (groups[prec].empty()) continue;
        waves_of[prec] = l2_waves(groups[prec], prec);
        // the block size that most of the staple kernel's sites are best served
        // by, unless the caller set one; a timing of one lattice counts only where
        // a launch is about that large (16 lattices of 4800 sites, FP64, 100 steps:
        // 18.6 ms with 384 threads, 22.5 with the 256 that suit one of them)
        long long votes[4] = {0, 0, 0, 0}, most = 0;
        for (const auto& wave : waves_of[prec]) {
            std::vector<const Geom*> g;
            for (const auto* r : wave) g.push_back(&r->buf.g);
            const StapleSites n = staple_sites(prec, g, ctx->sm_count);
            for (const long long sites : {n.one_sum, n.parts}) {
                votes[default_shape(prec, sites).threads / 128] += sites;
                most = std::max(most, sites);
            }
        }
        const bool like_one = 2 * most <= 3 * bigV;
        shapes[prec] = shape_for(ctx, prec, big, like_one);
        const StageChoice chosen = tuned_stage(ctx, prec, bigV);
        const int best = (int)(std::max_element(votes, votes + 4) - votes);
        if (votes[best] > 0 && (chosen == StageChoice::none || (chosen == StageChoice::timed && !like_one)))
            shapes[prec].threads = 128 * best;
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int launches = 0, rc = LGF_OK, threads_used = 0;
    cudaEventRecord(e0, ctx->stream);
    for (int prec = 0; prec < 2 && rc == LGF_OK; ++prec) {
        if (groups[prec].empty()) continue;
        threads_used = shapes[prec].threads;
        // one group for every wave of this precision, sized for the largest:
        // a wave replaces the previous one's members without a new group, a
        // new capture or a device synchronisation in between
        const auto& waves = waves_of[prec];
        long long max_tiles = 1;
        int max_members = 1;
        for (const auto& wave : waves) {
            long long t = 0;
            for (auto* r : wave) t += (4LL * r->buf.g.V + shapes[prec].threads - 1) / shapes[prec].threads;
            max_tiles = std::max(max_tiles, t);
            max_members = std::max(max_members, (int)wave.size());
        }
        std::unique_ptr<GroupBase> grp(make_group(ctx, prec, shapes[prec], max_members, max_tiles, true, true,
                                                  std::min(max_members, 32)));
        if (!grp) {
            rc = ctx->err.empty() ? set_error(ctx, LGF_ENOMEM, "group creation failed") : LGF_ECUDA;
            break;
        }
        for (auto wave : waves) {
            rc = run_wave(ctx, prec, wave, grp.get(), &launches);
            if (rc != LGF_OK) break;
        }
    }
    cudaEventRecord(e1, ctx->stream);
    cudaError_t e = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (e == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc == LGF_OK && e != cudaSuccess) rc = set_error(ctx, LGF_ECUDA, "batch failed: %s", cudaGetErrorString(e));
    if (rc == LGF_OK) rc = fetch_results(ctx, runs);
    if (stats) {
        stats->seconds = ms * 1e-3;
        stats->site_steps = site_steps;
        stats->launches = launches;
        stats->block_threads = threads_used;
    }
    cleanup();
    return rc;
}

}  // extern "C"
