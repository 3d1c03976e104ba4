// gfc_noalloc.cu -- e2 and theta of caller-owned device links with no device
// allocation.
//
// Who needs this: a caller whose device memory is entirely owned by something
// else -- a serving process whose allocator has carved up the whole GPU, or an
// application that sizes every buffer up front -- and a caller that shares the GPU
// with latency-sensitive work on other streams.  Such callers cannot let the
// library call cudaMalloc/cudaFree: an allocation can fail or fragment the
// caller's pool, and cudaFree synchronises the whole device, stalling everyone
// else's streams.  The context API (gfc_ctx_*) allocates its own scratch, so it
// is unusable for them; this entry point takes the links where the caller keeps
// them and uses a fixed scratch array compiled into the library instead.
//
// The scratch is a file-scope __device__ array of GFC_NOALLOC_SCRATCH_DOUBLES
// doubles (128 KiB).  Every GPU that loads the library holds one copy until the
// process exits.  All calls on a GPU share it and it keeps the contents of the
// last call, so two calls whose kernels overlap on the GPU (e.g. issued on two
// streams) race on it and give wrong results: serialise them.  Nothing in it needs
// to start at zero -- each call writes every slot it later reads.
//
// The first call on each device looks up the array's device address
// (cudaGetSymbolAddress) with that device current and caches it.  Every call is
// synchronous: it copies its two sums back to the host and waits for them on
// `stream` before returning.
//
// The links must be device memory of the current device (or managed memory):
// cudaPointerGetAttributes, which allocates nothing, is asked first, and pageable
// or page-locked host memory and another GPU's memory are refused before any
// kernel is launched.
#include <mutex>

#include "gfc.h"
#include "gfc_ctx.h"
#include "gfc_device.cuh"
#include "gfc_internal.h"
#include "gfc_reduce.cuh"

namespace gfc {

static __device__ __align__(256) double g_noalloc_scratch[GFC_NOALLOC_SCRATCH_DOUBLES];

namespace {

constexpr int NA_BLOCK = 64, NA_MIN_BLOCKS = 8;   // k_obs_partials_noalloc
constexpr int NA_FIN_BLOCK = 256;                  // k_finalize_noalloc
constexpr int NA_MAX_DEVICES = 64;
std::mutex na_mutex;
double *na_scratch[NA_MAX_DEVICES] = {nullptr};

__device__ __forceinline__ void na_load_aos(const double2 *__restrict__ u, uint32_t L, int mu, M3 &m) {
    const double2 *p = u + ((size_t)L * 4 + mu) * 9;
#pragma unroll
    for (int c = 0; c < 9; c++) m.e[c] = p[c];
}

// e2 density (sum of the 8 algebra components squared, gauge_fixing.c:428-438)
// and theta density (Re Tr divA divA^dagger, gauge_fixing.c:374-380) of site L
__device__ __forceinline__ void na_site(const double2 *__restrict__ u, const Lat &l, uint32_t L, double &e2,
                                        double &th) {
    Coord c = coord_lex(l, L);
    DivA dA;
    diva_zero(dA);
#pragma unroll
    for (int d = 0; d < 3; d++) {
        M3 f, r;
        na_load_aos(u, L, d + 1, f);
        na_load_aos(u, back_L(l, c, d), d + 1, r);
        diva_add(dA, f, r);
    }
    diva_densities(dA, e2, th);
}

// grid (nbx, nt): block bx of timeslice t writes scratch[(t*nbx + bx)*2 + {0,1}].  Bound by
// the latency and the tags of its loads: lanes lie 576 bytes apart, so each of a site's 54
// loads touches 32 lines.  So what counts is warps in flight: with DivA's 9 sums instead
// of whole matrices 128 registers do (16 warps per SM), and blocks of two warps, up to two
// rounds of them, leave the shortest last wave.  A call, copy and synchronisation
// included, at 8^3 x 16 / 16^3 x 32 / 24^3 x 48 / 32^3 x 64: 20.1 / 45.4 / 132 / 336 us;
// 128-thread blocks 22.8 / 44.4 / 132 / 361, at 166 registers 21.9 / 47.1 / 133 / 370;
// 256-thread blocks on whole matrices 30.7 / 56.0 / 147 / 377.
__global__ void __launch_bounds__(NA_BLOCK, NA_MIN_BLOCKS) k_obs_partials_noalloc(const double2 *__restrict__ u,
                                                                                  Lat l,
                                                                                  double *__restrict__ scratch) {
    __shared__ double sh[2][NA_BLOCK / 32];
    grid_wait();
    const uint32_t t = blockIdx.y;
    double v0 = 0.0, v1 = 0.0;
    for (uint32_t k = blockIdx.x * NA_BLOCK + threadIdx.x; k < l.vs; k += gridDim.x * NA_BLOCK) {
        double e2, th;
        na_site(u, l, t * l.vs + k, e2, th);
        v0 += e2;
        v1 += th;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v0 += __shfl_down_sync(0xffffffffu, v0, o);
        v1 += __shfl_down_sync(0xffffffffu, v1, o);
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
        sh[0][wid] = v0;
        sh[1][wid] = v1;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s0 = 0.0, s1 = 0.0;
        for (int w = 0; w < NA_BLOCK / 32; w++) {
            s0 += sh[0][w];
            s1 += sh[1][w];
        }
        size_t o = ((size_t)t * gridDim.x + blockIdx.x) * 2;
        scratch[o] = s0;
        scratch[o + 1] = s1;
    }
}

// one block (launch_early): sums the nparts partial pairs in index order into scratch[res_off + {0,1}]
__global__ void __launch_bounds__(NA_FIN_BLOCK) k_finalize_noalloc(double *__restrict__ scratch, uint32_t nparts,
                                                                   uint32_t res_off) {
    grid_wait();
    __shared__ double acc[2][NA_FIN_BLOCK];
    double s0 = 0.0, s1 = 0.0;
    for (uint32_t p = threadIdx.x; p < nparts; p += NA_FIN_BLOCK) {
        s0 += scratch[2 * (size_t)p];
        s1 += scratch[2 * (size_t)p + 1];
    }
    acc[0][threadIdx.x] = s0;
    acc[1][threadIdx.x] = s1;
    __syncthreads();
    for (int w = NA_FIN_BLOCK / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            acc[0][threadIdx.x] += acc[0][threadIdx.x + w];
            acc[1][threadIdx.x] += acc[1][threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        scratch[res_off] = acc[0][0];
        scratch[res_off + 1] = acc[1][0];
    }
}

// device address of the scratch array on the current device, looked up once
int na_scratch_ptr(double **out) {
    int dev = -1;
    GFC_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= NA_MAX_DEVICES) {
        set_error("gfc_e2_theta_device_noalloc: device ordinal %d outside 0..%d", dev, NA_MAX_DEVICES - 1);
        return GFC_ERR_ARG;
    }
    std::lock_guard<std::mutex> lock(na_mutex);
    if (!na_scratch[dev]) {
        double *p = nullptr;
        GFC_CHECK(cudaGetSymbolAddress((void **)&p, g_noalloc_scratch));
        na_scratch[dev] = p;
    }
    *out = na_scratch[dev];
    return GFC_OK;
}

}  // namespace
}  // namespace gfc

using namespace gfc;

extern "C" int gfc_e2_theta_device_noalloc(int ns, int nt, const double *u_dev, void *stream, double *e2,
                                           double *theta) {
    if (ns <= 0 || nt <= 0 || !u_dev || !e2 || !theta) {
        set_error("gfc_e2_theta_device_noalloc: bad arguments");
        return GFC_ERR_ARG;
    }
    if ((uintptr_t)u_dev % 16) {
        set_error("gfc_e2_theta_device_noalloc: u_dev must be 16-byte aligned (complex doubles are read in pairs)");
        return GFC_ERR_ARG;
    }
    {
        int cur = -1;
        GFC_CHECK(cudaGetDevice(&cur));
        cudaPointerAttributes pa;
        const cudaError_t pe = cudaPointerGetAttributes(&pa, u_dev);
        if (pe != cudaSuccess) {
            (void)cudaGetLastError();
            set_error("gfc_e2_theta_device_noalloc: u_dev is not a pointer the CUDA runtime knows (%s)",
                      cudaGetErrorString(pe));
            return GFC_ERR_ARG;
        }
        const bool ok = pa.type == cudaMemoryTypeManaged || (pa.type == cudaMemoryTypeDevice && pa.device == cur);
        if (!ok) {
            set_error("gfc_e2_theta_device_noalloc: u_dev must be device memory of the current device %d "
                      "(it is %s memory of device %d)", cur,
                      pa.type == cudaMemoryTypeHost ? "page-locked host"
                      : pa.type == cudaMemoryTypeDevice ? "device" : "unregistered host", pa.device);
            return GFC_ERR_ARG;
        }
    }
    const uint64_t V = (uint64_t)ns * ns * ns * nt;
    if (V * 4 >= (1ull << 31)) {
        set_error("gfc_e2_theta_device_noalloc: lattice %d^3x%d too large for 32-bit site indices", ns, nt);
        return GFC_ERR_GEOMETRY;
    }
    const Lat l = make_lat(ns, nt);
    uint32_t nbx = (l.vs + NA_BLOCK - 1) / NA_BLOCK;
    const uint32_t want = (2u * NA_MIN_BLOCKS * 148u + (uint32_t)nt - 1) / (uint32_t)nt;
    if (nbx > want) nbx = want;
    if (nbx < 1) nbx = 1;
    const uint64_t nparts = (uint64_t)nbx * (uint64_t)nt;
    const uint64_t res_off = ((2 * nparts + 31) / 32) * 32;   // keep the result 256-byte aligned
    if (res_off + 2 > GFC_NOALLOC_SCRATCH_DOUBLES) {
        set_error("gfc_e2_theta_device_noalloc: nt=%d needs %llu scratch doubles, the fixed scratch holds %d "
                  "(use gfc_ctx_e2 for this lattice)",
                  nt, (unsigned long long)(res_off + 2), GFC_NOALLOC_SCRATCH_DOUBLES);
        return GFC_ERR_ARG;
    }
    double *scratch = nullptr;
    int rc = na_scratch_ptr(&scratch);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    k_obs_partials_noalloc<<<dim3(nbx, nt), NA_BLOCK, 0, s>>>((const double2 *)u_dev, l, scratch);
    launch_early(k_finalize_noalloc, 1, NA_FIN_BLOCK, 0, s, scratch, (uint32_t)nparts, (uint32_t)res_off);
    GFC_CHECK(cudaGetLastError());
    double h[2];
    GFC_CHECK(cudaMemcpyAsync(h, scratch + res_off, sizeof h, cudaMemcpyDeviceToHost, s));
    GFC_CHECK(cudaStreamSynchronize(s));
    *e2 = h[0] / (double)V;
    *theta = h[1] / (3.0 * (double)V);
    return GFC_OK;
}
