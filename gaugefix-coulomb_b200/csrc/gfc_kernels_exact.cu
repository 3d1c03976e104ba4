// gfc_kernels_exact.cu -- FP64 kernels that round exactly like the reference.
//
// k_sweep_exact: one checkerboard half-sweep (gauge_fixing.c:773-787) over the sites
// of one parity, one thread per site.  Each thread builds w(x) from its 3 forward
// and 3 backward spatial links (calculate_w, gauge_fixing.c:445-531), computes the
// over-relaxed update with reference arithmetic (xor_update), and applies it to
// G(x), the 3 forward links and the 3 backward links (updateLocalUG,
// gauge_fixing.c:600-651).  With even ns no two sites of one parity share a link,
// so the parallel half-sweep equals the reference's sequential one bit for bit.
//
// Temporal links are not touched here: they never enter w, e2, theta or F, so
// their transformation is applied once at the end (k_temporal_transform).
//
// Memory traffic per site-update: 6 links + G read and written = 14 x 144 B.
#include <algorithm>

#include "gfc_device.cuh"
#include "gfc.h"
#include "gfc_ctx.h"
#include "gfc_internal.h"
#include "gfc_reduce.cuh"

namespace gfc {

template <bool CB>
__device__ __forceinline__ void site_update_exact(double2 *__restrict__ u, double2 *__restrict__ g,
                                                  const Lat &l, int par, const Coord &c, double omega,
                                                  unsigned hits) {
    const int op = CB ? (par ^ 1) : 0;
    const int sp = CB ? par : 0;
    const uint32_t si = CB ? (c.L >> 1) : c.L;
    uint32_t ib[3];
#pragma unroll
    for (int d = 0; d < 3; d++) ib[d] = CB ? (back_L(l, c, d) >> 1) : back_L(l, c, d);

    M3 w;
#pragma unroll
    for (int k = 0; k < 9; k++) w.e[k] = cz();
#pragma unroll
    for (int d = 0; d < 3; d++) {
        M3 f, r;
        load_m(u + uidx(l, d, sp, 0, si), l.vh, f);
        load_m(u + uidx(l, d, op, 0, ib[d]), l.vh, r);
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 3; b++)
                w.e[EL(a, b)] = xcadd(w.e[EL(a, b)], xcadd(f.e[EL(a, b)], cconj(r.e[EL(b, a)])));
    }

    M3 upd;
    xor_update(w, omega, hits, upd);

    M3 m, t;
    load_m(g + gidx(l, sp, 0, si), l.vh, m);
    xprod(upd, m, t);
    store_m(g + gidx(l, sp, 0, si), l.vh, t);
#pragma unroll
    for (int d = 0; d < 3; d++) {
        load_m(u + uidx(l, d, sp, 0, si), l.vh, m);
        xprod(upd, m, t);
        store_m(u + uidx(l, d, sp, 0, si), l.vh, t);
        load_m(u + uidx(l, d, op, 0, ib[d]), l.vh, m);
        xprod_dag(m, upd, t);
        store_m(u + uidx(l, d, op, 0, ib[d]), l.vh, t);
    }
}

// Launch shapes (threads per block, minimum resident blocks per SM); the second
// caps registers per thread.  gfc_ctx_autotune picks one per lattice.
// stop (may be null): a stop word set on the device; once it is, the launch does nothing
template <int BLOCK, int MINB>
__global__ void __launch_bounds__(BLOCK, MINB) k_sweep_exact(double2 *__restrict__ u, double2 *__restrict__ g,
                                                             Lat l, int par, double omega, unsigned hits,
                                                             const unsigned *stop) {
    grid_wait();
    if (stop && *(volatile const unsigned *)stop) return;
    uint32_t i = blockIdx.x * BLOCK + threadIdx.x;
    if (i >= l.vh) return;
    Coord c = coord_cb(l, par, i);
    site_update_exact<true>(u, g, l, par, c, omega, hits);
}

// The same update with the six links first copied into shared memory by cp.async
// (9 x 16 B per link per thread: the whole site's links requested at once, no
// registers held for them), read back from there for the link update instead of
// being loaded again.  Arithmetic and order are those of site_update_exact.
// Staged layout: entry e of link m of thread x at sm[(m * 9 + e) * BLOCK + x],
// m = 2d forward, 2d+1 backward link of direction d.  CB = false: the lexicographic
// layout of odd ns (one parity slot, slot index = the site's lexicographic index).
template <int BLOCK, bool CB = true>
__device__ __forceinline__ void site_update_exact_staged(double2 *__restrict__ u, double2 *__restrict__ g,
                                                         const Lat &l, int par, const Coord &c, double omega,
                                                         unsigned hits, double2 *sm) {
    if (!CB) par = 0;
    const int op = CB ? par ^ 1 : 0;
    const uint32_t si = CB ? c.L >> 1 : c.L;
    // G is read only after the update is known: ask for it in L2 now
#pragma unroll
    for (int e = 0; e < 9; e++) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(g + gidx(l, par, e, si)));
    uint32_t ib[3];
#pragma unroll
    for (int d = 0; d < 3; d++) ib[d] = CB ? back_L(l, c, d) >> 1 : back_L(l, c, d);
    double2 *my = sm + threadIdx.x;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const double2 *f = u + uidx(l, d, par, 0, si);
        const double2 *r = u + uidx(l, d, op, 0, ib[d]);
#pragma unroll
        for (int e = 0; e < 9; e++) {
            const unsigned sf = (unsigned)__cvta_generic_to_shared(my + ((2 * d) * 9 + e) * BLOCK);
            const unsigned sr = (unsigned)__cvta_generic_to_shared(my + ((2 * d + 1) * 9 + e) * BLOCK);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sf), "l"(f + (size_t)e * l.vh) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sr), "l"(r + (size_t)e * l.vh) : "memory");
        }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");

    // The direction loops stay rolled: one copy of each body keeps the kernel within
    // the instruction cache (the operands come from shared memory, so no load
    // parallelism is lost); the arithmetic and its order are unchanged.
    M3 w;
#pragma unroll
    for (int k = 0; k < 9; k++) w.e[k] = cz();
#pragma unroll 1
    for (int d = 0; d < 3; d++) {
        M3 f, r;
        load_m(my + (2 * d) * 9 * BLOCK, BLOCK, f);
        load_m(my + (2 * d + 1) * 9 * BLOCK, BLOCK, r);
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 3; b++)
                w.e[EL(a, b)] = xcadd(w.e[EL(a, b)], xcadd(f.e[EL(a, b)], cconj(r.e[EL(b, a)])));
    }

    M3 upd;
    xor_update(w, omega, hits, upd);
    asm volatile("" ::: "memory");   // read the links again from shared memory below

    // G is loaded here and multiplied after the six link updates, which hide its
    // latency (the products are independent, so their order changes no result)
    M3 m, t, gm;
    load_m(g + gidx(l, par, 0, si), l.vh, gm);
#pragma unroll 1
    for (int d = 0; d < 3; d++) {
        const uint32_t b = d == 0 ? ib[0] : (d == 1 ? ib[1] : ib[2]);
        load_m(my + (2 * d) * 9 * BLOCK, BLOCK, m);
        xprod(upd, m, t);
        store_m(u + uidx(l, d, par, 0, si), l.vh, t);
        load_m(my + (2 * d + 1) * 9 * BLOCK, BLOCK, m);
        xprod_dag(m, upd, t);
        store_m(u + uidx(l, d, op, 0, b), l.vh, t);
    }
    xprod(upd, gm, t);
    store_m(g + gidx(l, par, 0, si), l.vh, t);
}

template <int BLOCK, int MINB>
__global__ void __launch_bounds__(BLOCK, MINB) k_sweep_exact_staged(double2 *__restrict__ u,
                                                                    double2 *__restrict__ g, Lat l, int par,
                                                                    double omega, unsigned hits,
                                                                    const unsigned *stop) {
    extern __shared__ __align__(16) unsigned char exact_stage[];
    grid_wait();
    if (stop && *(volatile const unsigned *)stop) return;
    uint32_t i = blockIdx.x * BLOCK + threadIdx.x;
    if (i >= l.vh) return;
    Coord c = coord_cb(l, par, i);
    site_update_exact_staged<BLOCK>(u, g, l, par, c, omega, hits, (double2 *)exact_stage);
}

template <int BLOCK, int MINB>
static void launch_exact_staged(const Lat &l, double2 *u, double2 *g, int par, double omega, unsigned hits,
                                cudaStream_t s, const unsigned *stop) {
    constexpr size_t bytes = (size_t)6 * 9 * BLOCK * sizeof(double2);
    static_assert(bytes <= 227 * 1024, "staged links exceed shared memory");
    auto kern = k_sweep_exact_staged<BLOCK, MINB>;
    static std::atomic<unsigned long long> done{0};
    smem_attr_once(done, kern, bytes);
    launch_early(kern, (l.vh + BLOCK - 1) / BLOCK, BLOCK, bytes, s, u, g, l, par, omega, hits, stop);
}

// Odd ns: same-parity sites meet across the periodic boundary, so the updates of a
// half-sweep depend on their order; the reference visits a timeslice in z, y, x
// order (LOOP_SPATIAL).  Two sites of one parity share a link only across the
// boundary: a site with coordinate 0 in direction d and the one with ns - 1 there
// (other coordinates equal), and the reference always updates the first before the
// second.  Ordering the sites by their number of coordinates equal to ns - 1 (the
// boundary level, 0..3) therefore puts every such pair in consecutive levels, in
// the reference's order, and no two sites of one level share a link: sweeping
// level 0, then 1, 2 and 3, each level in parallel, gives every site the links the
// sequential sweep gives it, bit for bit.  Lexicographic layout.
//
// The threads of a launch take the level's sites of the half-sweep's parity, numbered
// without gaps (odd_level_site), and stage the six links of a site in shared memory as
// the even-ns kernel does.  31^3 x 64: 847 us per half-sweep when every launch tested all
// sites of the parity for the level, 659 with this numbering; 15^3 x 32: 81 and 79.
constexpr int LEVEL_BLOCK = 32;
__global__ void __launch_bounds__(LEVEL_BLOCK, 8) k_sweep_exact_level(double2 *__restrict__ u,
                                                                     double2 *__restrict__ g, Lat l, int sweep,
                                                                     int level, double omega, unsigned hits,
                                                                     const unsigned *stop) {
    extern __shared__ __align__(16) unsigned char level_stage[];
    grid_wait();
    if (stop && *(volatile const unsigned *)stop) return;
    const uint32_t n = odd_level_count(l, level), k = blockIdx.x * LEVEL_BLOCK + threadIdx.x, t = k / n;
    uint32_t off;
    // BLACKRED_SWEEP (gauge_fixing.c:42): parity (x + y + z + t) & 1 = sweep & 1
    if (t >= (uint32_t)l.nt || !odd_level_site(l, sweep & 1, t, level, k - t * n, off)) return;
    Coord c = coord_lex(l, t * l.vs + off);
    // ns = 1: a site's forward and backward link in a direction are one link, updated
    // twice in turn (g U, then that times g^dagger); the unstaged form reads it again
    // between the two, the staged one would not
    if (l.ns == 1)
        site_update_exact<false>(u, g, l, 0, c, omega, hits);
    else
        site_update_exact_staged<LEVEL_BLOCK, false>(u, g, l, 0, c, omega, hits, (double2 *)level_stage);
}

// The same half-sweep in one launch, a warp to a piece (OddPieces): 15^3 x 32 53 us per
// half-sweep where the four launches take 79, 31^3 x 64 773 us where they take 660.
__global__ void __launch_bounds__(LEVEL_BLOCK, 8) k_sweep_exact_pieces(double2 *__restrict__ u,
                                                                      double2 *__restrict__ g, Lat l, int sweep,
                                                                      double omega, unsigned hits,
                                                                      const unsigned *stop) {
    extern __shared__ __align__(16) unsigned char level_stage[];
    grid_wait();
    if (stop && *(volatile const unsigned *)stop) return;
    uint32_t k = blockIdx.x / l.nt;   // the longest pieces (corners, edges) first
    const uint32_t t = blockIdx.x - k * l.nt;
    const int kind = OddPieces(l).kind(k);
#pragma unroll 1
    for (int level = 0; level <= 3 - kind; level++) {
        uint32_t off;
        if (odd_piece_site(l, sweep & 1, t, kind, k, threadIdx.x, level, off))
            site_update_exact_staged<LEVEL_BLOCK, false>(u, g, l, 0, coord_lex(l, t * l.vs + off), omega, hits,
                                                         (double2 *)level_stage);
        if (level < 3 - kind) odd_level_fence();
    }
}

int exact_num_shapes() { return 5; }

// returns the number of kernels launched
int launch_sweep_exact(double2 *u, double2 *g, const Lat &l, int sweep, double omega, unsigned hits,
                        cudaStream_t s, int shape, const unsigned *stop) {
    if (l.cb) {
        int par = sweep & 1;  // BLACKRED_SWEEP: even sites on even sweeps (gauge_fixing.c:42)
        switch (shape) {
            case 1:
                launch_early(k_sweep_exact<128, 3>, (l.vh + 127) / 128, 128, 0, s, u, g, l, par, omega, hits, stop);
                break;
            case 2:   // 27 KiB per CTA, 8 CTAs per SM
                launch_exact_staged<32, 8>(l, u, g, par, omega, hits, s, stop);
                break;
            case 3:   // 110.6 KiB of staged links per CTA, 2 CTAs per SM
                launch_exact_staged<128, 2>(l, u, g, par, omega, hits, s, stop);
                break;
            case 4:   // 55.3 KiB per CTA, 4 CTAs per SM
                launch_exact_staged<64, 4>(l, u, g, par, omega, hits, s, stop);
                break;

            default:
                launch_early(k_sweep_exact<128, 1>, (l.vh + 127) / 128, 128, 0, s, u, g, l, par, omega, hits, stop);
                break;
        }
    } else {
        constexpr size_t bytes = (size_t)6 * 9 * LEVEL_BLOCK * sizeof(double2);
        static std::atomic<unsigned long long> done{0};
        smem_attr_once(done, k_sweep_exact_level, bytes);
        // one launch up to two waves of its warps (8 per SM), where a launch is a warp's
        // chain of instructions; level by level where the sectors of whole rows count
        if (l.ns > 1 && OddPieces(l).count() * (uint32_t)l.nt <= 2 * 8 * 148) {
            static std::atomic<unsigned long long> done_p{0};
            smem_attr_once(done_p, k_sweep_exact_pieces, bytes);
            launch_early(k_sweep_exact_pieces, OddPieces(l).count() * l.nt, LEVEL_BLOCK, bytes, s, u, g, l, sweep,
                         omega, hits, stop);
            return 1;
        }
        int launched = 0;
        for (int level = l.ns == 1 ? 3 : 0; level < 4; level++, launched++)   // ns = 1: corners only
            launch_early(k_sweep_exact_level, (odd_level_count(l, level) * l.nt + LEVEL_BLOCK - 1) / LEVEL_BLOCK,
                         LEVEL_BLOCK, bytes, s, u, g, l, sweep, level, omega, hits, stop);
        return launched;
    }
    return 1;
}

// ----------------------------------------------------------- reunitarise --
// reunitarizeField (fields.c:144-187): projectSU3 on every matrix of nmat
// SoA matrices laid out as [c][stride] blocks starting at base + k*9*stride.
__global__ void k_reunitarize(double2 *__restrict__ base, uint32_t stride, uint32_t nblk,
                              unsigned *__restrict__ status) {
    grid_wait();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t k = blockIdx.y;
    if (i >= stride || k >= nblk) return;
    double2 *p = base + (size_t)k * 9 * stride + i;
    M3 m;
    load_m(p, stride, m);
    int st = xproject(m);
    store_m(p, stride, m);
    if (st) atomicOr(status, GFC_STATUS_PROJECT_FAIL);
}

void launch_reunitarize(double2 *base, uint32_t stride, uint32_t nblk, unsigned *status, cudaStream_t s) {
    dim3 grid((stride + 255) / 256, nblk);
    launch_early(k_reunitarize, grid, 256, 0, s, base, stride, nblk, status);
}

__global__ void k_identity(double2 *__restrict__ g, uint32_t n) {
    grid_wait();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
#pragma unroll
    for (int c = 0; c < 9; c++) g[(size_t)c * n + i] = make_double2((c % 4) == 0 ? 1.0 : 0.0, 0.0);
}

// G is npar blocks of [9][vh]; treat it as one [9][npar*vh] run per block
void launch_identity(double2 *g, const Lat &l, cudaStream_t s) {
    for (int p = 0; p < l.npar; p++)
        launch_early(k_identity, (l.vh + 255) / 256, 256, 0, s, g + (size_t)p * 9 * l.vh, l.vh);
}

// ------------------------------------------------------------- observables --
// Per site: div A (four_potential.c:70-113) -> e2 and theta densities (gfc_reduce.cuh);
// block partials per timeslice, summed by the last block.
template <bool CB>
__device__ __forceinline__ void site_obs(const double2 *__restrict__ u, const Lat &l, int par,
                                         const Coord &c, double &e2, double &th) {
    const int op = CB ? (par ^ 1) : 0;
    const int sp = CB ? par : 0;
    const uint32_t si = CB ? (c.L >> 1) : c.L;
    DivA dA;
    diva_zero(dA);
#pragma unroll
    for (int d = 0; d < 3; d++) {
        uint32_t Lb = back_L(l, c, d);
        uint32_t ib = CB ? (Lb >> 1) : Lb;
        M3 f, r;
        load_m(u + uidx(l, d, sp, 0, si), l.vh, f);
        load_m(u + uidx(l, d, op, 0, ib), l.vh, r);
        diva_add(dA, f, r);
    }
    diva_densities(dA, e2, th);
}

// grid (nbx, nt): block bx of slice t sums sites of both parities of slice t.  The
// parities alternate from thread to thread (k -> parity k & 1, slot k >> 1): a
// site's backward links are the other parity's, so they are read by a neighbouring
// thread or a recent block and come from L2, not a second time from DRAM, as they
// would if one parity's half of the slice were swept before the other's.
// The six links of a site are requested at once; 128-thread blocks, four to an SM.
// 32^3 x 64, call to call: 214 us with the reference's operations all carried out (1000
// FP64 operations per site, most of them scalings and mirror images, see DivA) and a
// second launch for the sums, 198 us now; its bytes take 139 us at the copy rate.  (223 us
// marching in z and passing a link's part on to the next site's thread: half the bytes
// from L2, but its loads wait for one another.)
//
// With stop (a stop word; once set, the launch does nothing) and sweep > 0 the proxy (e2 =
// out[0] / V, or theta = out[1] / 3V, normalised as the host does) below tol sets *stop
// to sweep: later sweep and observables launches of the stream then do nothing.
__global__ void __launch_bounds__(128, 4) k_obs(const double2 *__restrict__ u, Lat l, double *__restrict__ part,
                                                unsigned *__restrict__ ticket, double *__restrict__ out,
                                                double *__restrict__ slice_out, unsigned *stop, int theta, double tol,
                                                int sweep) {
    grid_wait();
    if (stop && *(volatile const unsigned *)stop) return;
    const uint32_t t = blockIdx.y;
    const uint32_t vsh = l.cb ? l.vs / 2 : l.vs;  // slots of one parity per slice
    const uint32_t n = vsh * l.npar;
    double v[2] = {0.0, 0.0};
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int par = l.cb ? (int)(k & 1u) : 0;
        const uint32_t i = t * vsh + (l.cb ? k >> 1 : k);
        double e2, th;
        if (l.cb) {
            Coord c = coord_cb(l, par, i);
            site_obs<true>(u, l, par, c, e2, th);
        } else {
            Coord c = coord_lex(l, i);
            site_obs<false>(u, l, 0, c, e2, th);
        }
        v[0] += e2;
        v[1] += th;
    }
    block_sum<2>(v);
    if (last_block_sum<2>(v, part, ticket, slice_out)) {
        out[0] = v[0];
        out[1] = v[1];
        if (stop && sweep > 0) {
            const double n3 = (double)l.v, res = theta ? v[1] / (3.0 * n3) : v[0] / n3;
            if (res <= tol) *stop = (unsigned)sweep;
        }
    }
}

// F density: Re Tr of the 3 spatial links at a site (calculateF, gauge_fixing.c:289-337)
__global__ void __launch_bounds__(256) k_functional(const double2 *__restrict__ u, Lat l,
                                                    double *__restrict__ part, unsigned *__restrict__ ticket,
                                                    double *__restrict__ out) {
    grid_wait();
    const uint32_t t = blockIdx.y;
    const uint32_t vsh = l.cb ? l.vs / 2 : l.vs;
    const uint32_t n = vsh * l.npar;
    double v[1] = {0.0};
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        int par = (int)(k / vsh);
        uint32_t i = t * vsh + (k % vsh);
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const double2 *p = u + uidx(l, d, par, 0, i);
            v[0] += (p[0].x + p[(size_t)4 * l.vh].x) + p[(size_t)8 * l.vh].x;
        }
    }
    block_sum<1>(v);
    if (last_block_sum<1>(v, part, ticket, nullptr)) out[0] = v[0];
}

int obs_blocks_per_slice(const Lat &l) {
    // blocks of 128 sites and more, twelve or so per SM: three or four of them are resident
    // at a time, so that the last round is a small part of the whole (four per SM left
    // the second round of two nearly empty)
    const uint32_t n = (l.vs + 127) / 128, want = (12u * 148u + (uint32_t)l.nt - 1) / (uint32_t)l.nt;
    return (int)std::min(n, want);
}

void launch_obs(const double2 *u, const Lat &l, double *part, unsigned *ticket, double *out, double *slice_out,
                cudaStream_t s, unsigned *stop, int theta, double tol, int sweep) {
    launch_early(k_obs, dim3(obs_blocks_per_slice(l), l.nt), 128, 0, s, u, l, part, ticket, out, slice_out, stop, theta,
                 tol, sweep);
}

void launch_functional(const double2 *u, const Lat &l, double *part, unsigned *ticket, double *out, cudaStream_t s) {
    launch_early(k_functional, dim3(obs_blocks_per_slice(l), l.nt), 256, 0, s, u, l, part, ticket, out);
}

}  // namespace gfc

// Architecture of the device code the runtime loaded for this library on `device`
// (cudaFuncGetAttributes of one of its kernels): binaryVersion 100 is sm_100 machine
// code, ptxVersion the virtual architecture it was compiled from.
extern "C" int gfc_device_code_version(int device, int *binary_version, int *ptx_version) {
    if (!binary_version || !ptx_version) {
        gfc::set_error("gfc_device_code_version: null output");
        return GFC_ERR_ARG;
    }
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return gfc::cuda_fail(e, "gfc_device_code_version: cudaSetDevice");
    cudaFuncAttributes a;
    e = cudaFuncGetAttributes(&a, gfc::k_identity);
    if (e != cudaSuccess) return gfc::cuda_fail(e, "gfc_device_code_version: cudaFuncGetAttributes");
    *binary_version = a.binaryVersion;
    *ptx_version = a.ptxVersion;
    return GFC_OK;
}

// Self-check of xdiv_shared against IEEE division: count pseudo-random (a, b) pairs,
// significands random or with many trailing zeros or all ones (exact quotients,
// near-ties, the divisors next below powers of two), exponents mostly within a
// factor 2^64 of one and otherwise anywhere (zeros, subnormals, infinities, NaNs).
namespace gfc {
__device__ __forceinline__ uint64_t div_mix(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}
__device__ double div_operand(uint64_t h, uint64_t form) {
    uint64_t m = h & 0xFFFFFFFFFFFFFULL, e;
    if (form % 5 == 0) m = 0xFFFFFFFFFFFFFULL;
    else if (form % 5 == 1) m = (m >> 30) << 30;
    if ((form >> 3) % 8 == 0) e = (h >> 52) & 0x7FF;          // anywhere
    else e = 1023 - 64 + ((h >> 52) & 127);
    return __longlong_as_double((long long)((h & 0x8000000000000000ULL) | (e << 52) | m));
}
__global__ void k_check_division(uint64_t seed, long long count, unsigned long long *bad) {
    unsigned long long nbad = 0;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < count;
         k += (long long)gridDim.x * blockDim.x) {
        const uint64_t h1 = div_mix(seed + 2 * (uint64_t)k), h2 = div_mix(h1 ^ 0x5851F42D4C957F2DULL);
        const uint64_t f = div_mix(h2);
        const double a = div_operand(h1, f), b = div_operand(h2, f >> 8);
        const double want = xd(a, b), got = xdiv_shared(a, b, xrcp(b), xdiv_in_range(b));
        nbad += __double_as_longlong(want) != __double_as_longlong(got);
    }
    if (nbad) atomicAdd(bad, nbad);
}
}  // namespace gfc

extern "C" int gfc_check_division(int device, unsigned long long seed, long long count,
                                  unsigned long long *mismatches) {
    if (!mismatches || count < 0) {
        gfc::set_error("gfc_check_division: null output or negative count");
        return GFC_ERR_ARG;
    }
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return gfc::cuda_fail(e, "gfc_check_division: cudaSetDevice");
    unsigned long long *d = nullptr;
    if ((e = cudaMalloc(&d, sizeof *d)) != cudaSuccess) return gfc::cuda_fail(e, "gfc_check_division: cudaMalloc");
    if ((e = cudaMemset(d, 0, sizeof *d)) == cudaSuccess) {
        gfc::k_check_division<<<148 * 8, 256>>>(seed, count, d);
        if ((e = cudaGetLastError()) == cudaSuccess && (e = cudaDeviceSynchronize()) == cudaSuccess)
            e = cudaMemcpy(mismatches, d, sizeof *d, cudaMemcpyDeviceToHost);
    }
    cudaFree(d);
    return e == cudaSuccess ? GFC_OK : gfc::cuda_fail(e, "gfc_check_division");
}
