// E/Q measurement that allocates nothing.
//
// Some callers cannot allocate device memory: code that holds every byte of
// the GPU in its own pool (a framework's caching allocator, a serving process
// that reserves its memory at start-up and forbids allocation afterwards) or
// a real-time loop that must not enter the driver's allocator.  They already
// have the configuration in device memory and a place for the result, and
// only need the measurement.  lgf_measure_noalloc serves them: the per-block
// partial sums that lgf_measure keeps in memory it allocates live here in one
// file-scope device array of fixed size instead.
//
// The scratch array is a host-side symbol: host code must not pass its name
// to a kernel (that would hand the kernel a host address).  Its device address
// is looked up once per device with cudaGetSymbolAddress, with that device
// current.  CUDA loads modules lazily by default, so that lookup is also what
// places the array in the GPU's memory: lgf_ctx_create does it for its device
// (noalloc_preload), and otherwise the first call made on a device does it.
// Callers that reserve the rest of the GPU's memory must therefore create a
// context or make one call first, and the first call should come before any
// stream capture.  Once loaded, a GPU holds the array (4 MiB + 4 KiB) until
// the process exits.  All calls on one GPU share it and it keeps the last
// call's contents: two calls that can run at the same time on the same GPU
// (different streams, different host threads) race on it, so the caller must
// order them.  Nothing in it has to start at zero: each call writes every
// entry it later reads.
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "lgf_engine.cuh"

namespace lgf {
namespace {

constexpr int NOALLOC_MAX_PARTIALS = 262144;  // (x0 slices) x (32-site chunks per slice)
constexpr int NOALLOC_MAX_SLICES = 256;       // x0 extent
constexpr int NOALLOC_MAX_DEVICES = 64;

static __device__ __align__(256) double2 g_noalloc_scratch[NOALLOC_MAX_PARTIALS + NOALLOC_MAX_SLICES];

std::mutex g_noalloc_mu;
double2* g_noalloc_addr[NOALLOC_MAX_DEVICES] = {};

// Grid (nchunk, N0), one 32-site tile per block: the one-launch measurement
// (measure_tile) reading the caller's file-order links in place.  The fixed
// scratch has no room for the loops' projections that lgf_measure.cuh shares
// between sites.  Bound by link loads (load_link_from<true>): 15 per plane and
// quadrant with shared paths instead of 40 for separate loops.  Products keep
// all three rows of the caller's matrices (the loops' error against extended
// precision is the separate loops', 1e-15 of a flowed charge profile; with the
// third row rebuilt it was 8e-15, and links 1e-7 off SU(3) moved E and Q by as
// much).  One B200, all launches on 32x16^3: 2.81 ms with separate loops, 1.33
// so (two-row products 1.20; with those, a 16-byte load per lane instead of
// lane pairs 1.40, links read by fours 1.24: the selects cost more than the
// lines they save).
__global__ void __launch_bounds__(MEAS_SITES * MEAS_WARPS, 1) k_noalloc_measure(const cplx<double>* __restrict__ L, Geom g,
                                                                               double2* __restrict__ partials) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    measure_tile<double, false, true>(reinterpret_cast<MeasSmem<double, true>*>(smem_raw), L, g, blockIdx.y, blockIdx.x, partials,
                                      gridDim.x, MeasSites{});
}

// one block per slice: fixed-order sums, then out = [E, Q, E_slice, Q_slice]
__global__ void __launch_bounds__(RED_THREADS) k_noalloc_slices(const double2* __restrict__ partials, int nchunk, Geom g,
                                                                double2* __restrict__ slice_sums, double* __restrict__ out) {
    __shared__ double se[RED_THREADS], sq[RED_THREADS];
    const int t = blockIdx.x;
    double e = 0.0, q = 0.0;
    for (int j = threadIdx.x; j < nchunk; j += RED_THREADS) {
        const double2 v = partials[t * nchunk + j];
        e += v.x;
        q += v.y;
    }
    se[threadIdx.x] = e;
    sq[threadIdx.x] = q;
    __syncthreads();
    for (int w = RED_THREADS / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            se[threadIdx.x] += se[threadIdx.x + w];
            sq[threadIdx.x] += sq[threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double inv4pi2 = 1.0 / (4.0 * 3.14159265358979323846 * 3.14159265358979323846);
        out[2 + t] = se[0] / (double)g.Vs;
        out[2 + g.n[0] + t] = sq[0] * inv4pi2;
        slice_sums[t] = make_double2(se[0], sq[0]);
    }
}

__global__ void __launch_bounds__(RED_THREADS) k_noalloc_total(const double2* __restrict__ slice_sums, Geom g,
                                                               double* __restrict__ out) {
    __shared__ double se[RED_THREADS], sq[RED_THREADS];
    double e = 0.0, q = 0.0;
    for (int j = threadIdx.x; j < g.n[0]; j += RED_THREADS) {
        e += slice_sums[j].x;
        q += slice_sums[j].y;
    }
    se[threadIdx.x] = e;
    sq[threadIdx.x] = q;
    __syncthreads();
    for (int w = RED_THREADS / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            se[threadIdx.x] += se[threadIdx.x + w];
            sq[threadIdx.x] += sq[threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double inv4pi2 = 1.0 / (4.0 * 3.14159265358979323846 * 3.14159265358979323846);
        out[0] = se[0] * (1.0 / (double)g.V);
        out[1] = sq[0] * inv4pi2;
    }
}

// device address of the scratch array on the current device (looked up once,
// with the measurement kernel's shared-memory limit raised there)
int noalloc_scratch(int dev, double2** out) {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            if (e != cudaSuccess) cudaGetLastError();  // this lookup's own error
            return LGF_ECUDA;
        }
        e = cudaFuncSetAttribute(k_noalloc_measure, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)measure_smem_bytes<double, true>());
        if (e != cudaSuccess) {
            cudaGetLastError();
            return LGF_ECUDA;
        }
        g_noalloc_addr[dev] = (double2*)p;
    }
    *out = g_noalloc_addr[dev];
    return LGF_OK;
}

}  // namespace

// Called by lgf_ctx_create with the context's device current: loads this
// file's module on that device (placing the scratch array) and caches its
// address, so the first measurement allocates nothing even under lazy loading.
int noalloc_preload(int dev) {
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return LGF_OK;  // such devices are served on first call
    double2* p = nullptr;
    return noalloc_scratch(dev, &p);
}

}  // namespace lgf

extern "C" int lgf_measure_noalloc(const double* links, const int shape[4], double* out, void* stream) {
    using namespace lgf;
    if (!links || !out || !valid_shape(shape)) return LGF_EINVAL;
    const Geom g = make_geom(shape);
    const int nchunk = (g.Vs + MEAS_SITES - 1) / MEAS_SITES;
    if (g.n[0] > NOALLOC_MAX_SLICES || (long long)nchunk * g.n[0] > NOALLOC_MAX_PARTIALS) return LGF_ETOOBIG;
    if (((uintptr_t)links % 16) != 0 || ((uintptr_t)out % 8) != 0) return LGF_EINVAL;
    // an error that earlier work left pending on this thread is the caller's:
    // report it without clearing it, and launch nothing
    if (cudaPeekAtLastError() != cudaSuccess) return LGF_ECUDA;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) return LGF_ECUDA;
    double2* scratch = nullptr;
    int rc = noalloc_scratch(dev, &scratch);
    if (rc != LGF_OK) return rc;
    double2* partials = scratch;
    double2* slice_sums = scratch + NOALLOC_MAX_PARTIALS;
    cudaStream_t st = (cudaStream_t)stream;
    k_noalloc_measure<<<dim3(nchunk, g.n[0]), dim3(MEAS_SITES, MEAS_WARPS), measure_smem_bytes<double, true>(), st>>>(
        (const cplx<double>*)links, g, partials);
    k_noalloc_slices<<<g.n[0], RED_THREADS, 0, st>>>(partials, nchunk, g, slice_sums, out);
    k_noalloc_total<<<1, RED_THREADS, 0, st>>>(slice_sums, g, out);
    // nothing was pending at entry, so an error now comes from these launches
    if (cudaGetLastError() != cudaSuccess) return LGF_ECUDA;
    return LGF_OK;
}
