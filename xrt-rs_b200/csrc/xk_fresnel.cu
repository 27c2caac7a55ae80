// 2-D Fresnel propagation (waves::fresnel::fresnel_propagate,
// src/waves/fresnel.rs:53-106) on B200:
//
//   U(x_ix, z_iz) = sum_j es_j exp(i a ((x_ix - x_j)^2 + (z_iz - z_j)^2)),  a = k / (2 d)
//
// over a regular nx x nz screen (index iz * nx + ix), k = E / CHBAR * 1e7.
//
// Two paths:
//
// * XK_PATH_F64: the reference's sum run directly in FP64, one thread per
//   screen point, rays staged through shared memory, the per-term operations
//   in the reference's order (explicitly rounded, no FMA contraction) and the
//   terms added in ray order.
//
// * XK_PATH_SEPARABLE: on a regular screen the Fresnel kernel factorises,
//       exp(i a r^2) = exp(i a (x_ix - x_j)^2) * exp(i a (z_iz - z_j)^2),
//   so U = Z diag(es) X^T is a complex matrix product with the ray index as
//   the contraction. As a real product with interleaved (re, im) columns,
//       C[iz][n(ix, c)] = sum_k A[iz][k] B[n(ix, c)][k],
//       A[iz][2j] = Re Z, A[iz][2j+1] = Im Z,
//       B[n(ix,0)][2j] = Re W, B[n(ix,0)][2j+1] = -Im W, B[n(ix,1)][2j] = Im W, B[n(ix,1)][2j+1] = Re W,
//   with W = es X / max|es| and, per 128-point block of x, the real parts in
//   its first 128 columns and the imaginary parts in the next 128:
//   n(ix, c) = 256 (ix / 128) + 128 c + ix % 128. One fused kernel computes
//   it on the tensor cores without ever writing A or B to memory: per block
//   of 32 rays, a stager warp writes the rays' split coordinates to a ring of
//   shared-memory buffers, eight producer warps form the CTA's A (128 z rows)
//   and B (128 x points, 256 rows) tiles from them, split each phasor into
//   f16 hi + lo parts and store them in shared memory in the
//   128-byte-swizzled K-major layout; one thread issues tcgen05.mma kind::f16 (f32 accumulation in tensor
//   memory) for A_hi B_hi + A_hi B_lo + A_lo B_hi, which keeps ~2^-21 of each
//   phasor; four epilogue warps drain the accumulator into an FP64 partial
//   every kFSeg ray blocks (the tensor cores' f32 accumulation error grows
//   with the number of accumulated blocks), alternating between two TMEM
//   accumulators so that draining overlaps the next segment. K-split partials
//   are added in FP64 in split order (results do not depend on scheduling).

#include <cuda_fp16.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <mutex>

#include "xk_ctx.cuh"
#include "xk_phasor.cuh"

namespace xk {
namespace {

using namespace phasor;

constexpr double kInv2Pi = 0.15915494309189533577;

// ---- shared pieces -----------------------------------------------------------

// x_i = lo + (hi - lo) * i / max(n - 1, 1), evaluated as the reference does
// (src/waves/fresnel.rs:70-75).
__global__ void coords_kernel(double lo, double hi, size_t n, double* __restrict__ out) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double den = (double)(n > 1 ? n - 1 : 1);
    out[i] = __dadd_rn(lo, __ddiv_rn(__dmul_rn(__dsub_rn(hi, lo), (double)i), den));
}

// ---- FP64 direct sum ---------------------------------------------------------

constexpr int kF64Threads = 256;

__global__ void __launch_bounds__(kF64Threads)
fresnel_f64_kernel(const double* __restrict__ rx, const double* __restrict__ rz,
                   const double* __restrict__ er, const double* __restrict__ ei, size_t n,
                   const double* __restrict__ xp, const double* __restrict__ zp, size_t nx,
                   size_t total, double pre, double* __restrict__ o_re, double* __restrict__ o_im) {
    __shared__ double sx[kF64Threads], sz[kF64Threads], sr[kF64Threads], si[kF64Threads];
    const size_t idx = blockIdx.x * (size_t)kF64Threads + threadIdx.x;
    const bool valid = idx < total;
    const size_t iz = valid ? idx / nx : 0, ix = valid ? idx - iz * nx : 0;
    const double px = valid ? xp[ix] : 0.0, pz = valid ? zp[iz] : 0.0;
    double s_re = 0.0, s_im = 0.0;
    for (size_t base = 0; base < n; base += kF64Threads) {
        const size_t j = base + threadIdx.x;
        if (j < n) {
            sx[threadIdx.x] = rx[j];
            sz[threadIdx.x] = rz[j];
            sr[threadIdx.x] = er[j];
            si[threadIdx.x] = ei[j];
        }
        __syncthreads();
        const int len = (int)min((size_t)kF64Threads, n - base);
        for (int t = 0; t < len; ++t) {
            // dx, dz, r2 = dx*dx + dz*dz, phase = (0, pre) * r2, exp of it,
            // es * phasor, sum += (src/waves/fresnel.rs:87-94).
            const double dx = __dsub_rn(px, sx[t]);
            const double dz = __dsub_rn(pz, sz[t]);
            const double r2 = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dz, dz));
            double sn, cs;
            sincos(__dmul_rn(pre, r2), &sn, &cs);
            const double a = sr[t], b = si[t];
            s_re = __dadd_rn(s_re, __dsub_rn(__dmul_rn(a, cs), __dmul_rn(b, sn)));
            s_im = __dadd_rn(s_im, __dadd_rn(__dmul_rn(a, sn), __dmul_rn(b, cs)));
        }
        __syncthreads();
    }
    if (valid) {
        o_re[idx] = s_re;
        o_im[idx] = s_im;
    }
}

// ---- fused separable product on the tensor cores --------------------------------

constexpr int kFStages = 2;
constexpr uint32_t kFA = 128 * 64 * 2;           // one A tile (hi or lo): 128 rows x 128 B
constexpr uint32_t kFB = 256 * 64 * 2;           // one B tile: 256 rows x 128 B
constexpr uint32_t kFStage = 2 * kFA + 2 * kFB;  // A_hi | A_lo | B_hi | B_lo
#ifndef XK_FRESNEL_PROD_WARPS
#define XK_FRESNEL_PROD_WARPS 8
#endif
#ifndef XK_FRESNEL_ROWS_PER
#define XK_FRESNEL_ROWS_PER 2
#endif
constexpr int kFProdThreads = 32 * XK_FRESNEL_PROD_WARPS;  // warps 5..
constexpr int kFRowsPer = XK_FRESNEL_ROWS_PER;             // A rows (and x points) per producer
constexpr int kFRowThreads = 128 / kFRowsPer;              // producers per ray group
constexpr int kFChunks = 8 / (kFProdThreads / kFRowThreads);  // 16-byte chunks per producer
static_assert(kFChunks * (kFProdThreads / kFRowThreads) == 8 && kFRowThreads % 32 == 0,
              "producers must tile the 128 rows x 8 chunks of a block");
constexpr int kFThreads = 32 + kFEpiThreads + kFProdThreads + 32;  // + the ray stager warp
// Ray staging (one block per ring buffer), per ray 8 floats: {z hi, x hi,
// z lo, x lo} and {frac(a z^2), frac(a x^2), es_re, es_im} (coordinates
// relative to the screen centre, amplitude scaled by 1 / max|es|).
constexpr int kFMinSplit = 10;                   // fewest ray blocks per K split
constexpr uint32_t kFRayBytes = kFRays * 32;
constexpr size_t kFSmem = 1024 + (size_t)kFStages * kFStage + kFRayBufs * kFRayBytes + kFEpiBytes + 256;

struct FusedArgs {
    const double *rx, *rz, *er, *ei;
    size_t n;
    int ray_blocks, splits;
    const double *xp, *zp;
    size_t nx, nz;
    double a_turns;    // k / (2 d) / (2 pi)
    double inv_scale;  // 1 / max|es|
    double ox, oz;     // origin of the phase split (screen centre)
    double* partial;   // [splits][m_pad][n_pad]
    int m_pad, n_pad;
    int* err;
    uint32_t wait_limit;  // polls of every bounded mbarrier wait
    uint32_t stall;       // test hook: extra arrivals stage 0's barrier waits for (never made)
};

// Epilogue role (warps 1..4): drains each finished accumulator segment into
// this CTA's 128 rows of the FP64 split partial; `arrive_empty(b)` releases
// accumulator b to the MMA issuer. Warp w reads TMEM lanes 32 (w % 4) .. + 31
// (rows qd*32 .. +31 of the tile); lane l owns row qd*32 + l. Per 16-column
// chunk the lane converts its values to FP64 in its shared-memory staging row
// and hands the row to a bulk copy: the first segment stores it, later ones
// add it to the partial at the memory side (FP64 add, round to nearest). A
// segment's operations complete before the next segment's start, so the
// partial is s0 + s1 + ... in segment order, independent of timing. `stage`:
// this warp's 32 staging rows.
template <class ArriveEmpty>
__device__ __forceinline__ void drain_role(const FusedArgs& g, int warp, int lane, int mt, int nt,
                                           int sp, int nseg, uint32_t tmem, uint64_t* acc_full,
                                           unsigned char* stage, volatile int* flag,
                                           ArriveEmpty arrive_empty) {
    using namespace sm100;
    const int qd = warp & 3;
    if (nseg == 0) {
        double* rows0 = g.partial + ((size_t)sp * g.m_pad + (size_t)mt * 128 + qd * 32) * g.n_pad +
                        (size_t)nt * kFN + lane;
        for (int rr = 0; rr < 32; ++rr)
            for (int c = 0; c < kFN; c += 32) rows0[(size_t)rr * g.n_pad + c] = 0.0;
        return;
    }
    double* grow = g.partial + ((size_t)sp * g.m_pad + (size_t)mt * 128 + qd * 32 + lane) * g.n_pad +
                   (size_t)nt * kFN;
    unsigned char* srow = stage + lane * kFEpiRow;
    const uint32_t s_addr = smem_u32(srow);
    for (int q = 0; q < nseg; ++q) {
        const int b = q & 1;
        const bool ok = mbar_wait(&acc_full[b], (uint32_t)(q >> 1) & 1u, g.wait_limit);
        if (!__all_sync(0xffffffffu, ok)) {
            *flag = 1;
            break;
        }
        tc_fence_after();
        bulk_wait_all();  // the previous segment's writes to these rows are performed
#pragma unroll 1
        for (int c = 0; c < kFN / 16; ++c) {
            float v[16];
            tmem_ld_16cols(tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)(b * kFN + c * 16), v);
            bulk_wait_read();  // the staging row is free again
#pragma unroll
            for (int k = 0; k < 8; ++k)
                reinterpret_cast<double2*>(srow)[k] =
                    make_double2((double)v[2 * k], (double)v[2 * k + 1]);
            fence_proxy_async();
            if (q == 0)
                bulk_s2g(grow + c * 16, s_addr, 128);
            else
                bulk_add_s2g_f64(grow + c * 16, s_addr, 128);
            bulk_commit();
        }
        tc_fence_before();
        arrive_empty(b);
    }
    bulk_wait_all();
}

// Ray stager role (one warp): stages the ray blocks rb0 .. rb0 + nrb - 1 in a
// ring of kFRayBufs shared-memory buffers.
__device__ __forceinline__ void stage_rays_role(const FusedArgs& g, int lane, int rb0, int nrb,
                                                unsigned char* rays_smem, uint64_t* ray_full,
                                                uint64_t* ray_empty, volatile int* flag) {
    using namespace sm100;
    // Ray stager: lane l stages ray l of each block as (z, x) pairs for
    // the packed phase: {zh, xh, zl, xl}, {zf, xf, es_re, es_im}
    // (coordinates relative to the screen centre, amplitude scaled). The
    // next block's loads are in flight while the stager waits for its
    // buffer to be released.
    for (int i = 0; i < nrb; ++i) {
        const int rb = i % kFRayBufs;
        const size_t j = (size_t)(rb0 + i) * kFRays + lane;
        double x = g.ox, z = g.oz, er = 0.0, ei = 0.0;
        if (j < g.n) {
            x = __ldg(g.rx + j);
            z = __ldg(g.rz + j);
            er = __ldg(g.er + j);
            ei = __ldg(g.ei + j);
        }
        const bool ok = i < kFRayBufs || mbar_wait(&ray_empty[rb],
                                                   (uint32_t)(i / kFRayBufs - 1) & 1u, g.wait_limit);
        if (!__all_sync(0xffffffffu, ok)) {
            *flag = 1;
            return;
        }
        float xh, xl, xf, zh, zl, zf;
        split_coord(x - g.ox, g.a_turns, &xh, &xl, &xf);
        split_coord(z - g.oz, g.a_turns, &zh, &zl, &zf);
        float4* st = reinterpret_cast<float4*>(rays_smem + rb * kFRayBytes);
        st[2 * lane] = make_float4(zh, xh, zl, xl);
        st[2 * lane + 1] = make_float4(zf, xf, (float)(er * g.inv_scale), (float)(ei * g.inv_scale));
        __syncwarp();
        if (lane == 0) mbar_arrive(&ray_full[rb]);
    }
}

__global__ void __launch_bounds__(kFThreads, 1) fresnel_fused_kernel(FusedArgs g) {
    using namespace sm100;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(tiles + kFStages * kFStage);
    uint64_t* empty = full + kFStages;
    uint64_t* acc_full = empty + kFStages;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* ray_full = acc_empty + 2;
    uint64_t* ray_empty = ray_full + kFRayBufs;
    uint64_t* mma_done = ray_empty + kFRayBufs;  // every issued MMA has completed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
    volatile int* flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    unsigned char* rays_smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(tmem_slot) + 64 + 15) & ~static_cast<uintptr_t>(15));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int mt = blockIdx.x, nt = blockIdx.y, sp = blockIdx.z;
    const int rb0 = (int)((long long)g.ray_blocks * sp / g.splits);
    const int rb1 = (int)((long long)g.ray_blocks * (sp + 1) / g.splits);
    const int nrb = rb1 - rb0;
    const int nseg = (nrb + kFSeg - 1) / kFSeg;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kFStages; ++s) {
            mbar_init(&full[s], kFProdThreads / 32 + (s == 0 ? g.stall : 0u));  // per producer warp
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], kFEpiThreads);
        }
        for (int b = 0; b < kFRayBufs; ++b) {
            mbar_init(&ray_full[b], 1);                      // the stager warp
            mbar_init(&ray_empty[b], kFProdThreads / 32);  // one arrival per producer warp
        }
        mbar_init(mma_done, 1);
        mbar_init_fence();
        *flag = 0;
    }
    if (warp == 0) tmem_alloc(tmem_slot, 2 * kFN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // UMMA issuer: per ray block three K blocks (hi.hi, hi.lo, lo.hi);
            // segment q accumulates into buffer q & 1.
            constexpr uint32_t idesc = idesc_f16_f32(128, kFN);
            bool good = true;
            for (int q = 0; q < nseg && good; ++q) {
                const int b = q & 1, use = q >> 1;
                if (use >= 1 && !mbar_wait(&acc_empty[b], (uint32_t)(use - 1) & 1u, g.wait_limit)) {
                    *flag = 1;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem + (uint32_t)(b * kFN);
                const int i0 = q * kFSeg, i1 = min(nrb, i0 + kFSeg);
                for (int i = i0; i < i1; ++i) {
                    const int s = i % kFStages;
                    if (!mbar_wait(&full[s], (uint32_t)(i / kFStages) & 1u, g.wait_limit)) {
                        *flag = 1;
                        good = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a_hi = smem_u32(tiles + (size_t)s * kFStage);
                    const uint32_t a_lo = a_hi + kFA, b_hi = a_hi + 2 * kFA, b_lo = b_hi + kFB;
                    const uint32_t as[3] = {a_hi, a_hi, a_lo}, bs[3] = {b_hi, b_lo, b_hi};
#pragma unroll
                    for (int p = 0; p < 3; ++p)
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_f16(d, desc_kmajor_sw128(as[p] + 32u * k),
                                     desc_kmajor_sw128(bs[p] + 32u * k), idesc,
                                     (uint32_t)((i - i0) | p | k));
                    umma_commit(&empty[s]);
                }
                umma_commit(&acc_full[b]);
            }
            // A loop that gave up on a wait may leave MMAs in flight: wait
            // (bounded) for them before the accumulators are freed.
            umma_commit(mma_done);
            if (!mbar_wait(mma_done, 0, max(g.wait_limit, kMmaDrainPolls))) *flag = 1;
        }
        __syncwarp();
    } else if (warp <= 4) {
        unsigned char* tb = rays_smem + kFRayBufs * kFRayBytes + (warp - 1) * 32 * kFEpiRow;
        drain_role(g, warp, lane, mt, nt, sp, nseg, tmem, acc_full, tb, flag,
                   [&](int b) { mbar_arrive(&acc_empty[b]); });
    } else if (warp < 5 + kFProdThreads / 32) {
        // Producers: thread p owns kFRowsPer A rows r_k = (p % kFRowThreads) +
        // kFRowThreads k (screen z index mt*128 + r_k) and the B rows r_k,
        // 128 + r_k (screen x index nt*128 + r_k), for the 16-byte chunks
        // kFChunks q .. kFChunks (q + 1) - 1 (q = p / kFRowThreads) of each
        // ray block: every staged ray value a thread reads serves kFRowsPer
        // rows, and each store instruction of a warp covers 32 consecutive
        // rows. The stager warp stages each block's rays in shared memory up
        // to kFRayBufs blocks ahead.
        const int p = threadIdx.x - 160;
        const int q = p / kFRowThreads, rq = p % kFRowThreads;
        bool va[kFRowsPer], vb[kFRowsPer];
        // Per-row terms: kappa = -2 a p (hi, lo) and P = frac(a p^2), the A
        // row in .x and the B row in .y.
        float2 kh2[kFRowsPer], khn2[kFRowsPer], kl2[kFRowsPer], pp2[kFRowsPer];
#pragma unroll
        for (int k = 0; k < kFRowsPer; ++k) {
            const int r = rq + kFRowThreads * k;
            const size_t iz = (size_t)mt * 128 + r, ix = (size_t)nt * 128 + r;
            va[k] = iz < g.nz;
            vb[k] = ix < g.nx;
            const double zr = va[k] ? g.zp[iz] - g.oz : 0.0, xr = vb[k] ? g.xp[ix] - g.ox : 0.0;
            float kzh, kzl, kxh, kxl, pz, px, unused, h0, l0;
            split_coord(-2.0 * g.a_turns * zr, 0.0, &kzh, &kzl, &unused);
            split_coord(-2.0 * g.a_turns * xr, 0.0, &kxh, &kxl, &unused);
            split_coord(zr, g.a_turns, &h0, &l0, &pz);
            split_coord(xr, g.a_turns, &h0, &l0, &px);
            kh2[k] = make_float2(kzh, kxh);
            khn2[k] = make_float2(-kzh, -kxh);
            kl2[k] = make_float2(kzl, kxl);
            pp2[k] = make_float2(pz, px);
        }
        for (int i = 0; i < nrb; ++i) {
            const int s = i % kFStages, rb = i % kFRayBufs;
            bool ok = mbar_wait(&ray_full[rb], (uint32_t)(i / kFRayBufs) & 1u, g.wait_limit);
            ok = ok && mbar_wait(&empty[s], ((uint32_t)(i / kFStages) & 1u) ^ 1u, g.wait_limit);
            if (!__all_sync(0xffffffffu, ok)) {
                *flag = 1;
                break;
            }
            unsigned char* base = tiles + (size_t)s * kFStage;
            const float4* sr = reinterpret_cast<const float4*>(rays_smem + rb * kFRayBytes);
#pragma unroll 1
            for (int cc = 0; cc < kFChunks; ++cc) {
                const int c = kFChunks * q + cc;
                uint32_t ah[kFRowsPer][4], al[kFRowsPer][4], bh[kFRowsPer][4], bl[kFRowsPer][4];
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    const int j = 4 * c + jj;
                    const float4 v0 = sr[2 * j], v1 = sr[2 * j + 1];
#pragma unroll
                    for (int k = 0; k < kFRowsPer; ++k) {
                        // Phase in turns of the A row (.x) and the B row (.y).
                        const float2 t = pair_turns2(kh2[k], khn2[k], kl2[k],
                                                     __fadd2_rn(pp2[k], make_float2(v1.x, v1.y)),
                                                     make_float2(v0.x, v0.y),
                                                     make_float2(v0.z, v0.w));
                        const float2 th = __fmul2_rn(t, f2(6.28318530717958647692f));
                        float ca, sa, cb, sb, wr = 0.f, wi = 0.f;
                        __sincosf(th.x, &sa, &ca);
                        __sincosf(th.y, &sb, &cb);
                        if (!va[k]) ca = sa = 0.f;
                        if (vb[k]) {
                            wr = cmul_re(v1.z, v1.w, cb, sb);
                            wi = cmul_im(v1.z, v1.w, cb, sb);
                        }
                        split16x2(ca, sa, &ah[k][jj], &al[k][jj]);
                        split16x2(wr, wi, &bh[k][jj], &bl[k][jj]);
                    }
                }
                unsigned char* bhi = base + 2 * kFA;
                unsigned char* blo = bhi + kFB;
#pragma unroll
                for (int k = 0; k < kFRowsPer; ++k) {
                    const uint32_t r = (uint32_t)(rq + kFRowThreads * k);
                    // A row: (Re Z, Im Z); B rows r: (Re W, -Im W), 128 + r:
                    // (Im W, Re W). Each store instruction writes 32
                    // consecutive rows, which meet all eight swizzle phases
                    // (no bank conflict).
                    *reinterpret_cast<uint4*>(base + sw128(r, c)) =
                        make_uint4(ah[k][0], ah[k][1], ah[k][2], ah[k][3]);
                    *reinterpret_cast<uint4*>(base + kFA + sw128(r, c)) =
                        make_uint4(al[k][0], al[k][1], al[k][2], al[k][3]);
                    *reinterpret_cast<uint4*>(bhi + sw128(r, c)) =
                        make_uint4(neg_hi(bh[k][0]), neg_hi(bh[k][1]), neg_hi(bh[k][2]), neg_hi(bh[k][3]));
                    *reinterpret_cast<uint4*>(bhi + sw128(128 + r, c)) =
                        make_uint4(swap_halves(bh[k][0]), swap_halves(bh[k][1]),
                                   swap_halves(bh[k][2]), swap_halves(bh[k][3]));
                    *reinterpret_cast<uint4*>(blo + sw128(r, c)) =
                        make_uint4(neg_hi(bl[k][0]), neg_hi(bl[k][1]), neg_hi(bl[k][2]), neg_hi(bl[k][3]));
                    *reinterpret_cast<uint4*>(blo + sw128(128 + r, c)) =
                        make_uint4(swap_halves(bl[k][0]), swap_halves(bl[k][1]),
                                   swap_halves(bl[k][2]), swap_halves(bl[k][3]));
                }
            }
            // Make the generic-proxy stores visible to the tensor cores, then
            // one arrival per warp.
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&full[s]);
                mbar_arrive(&ray_empty[rb]);
            }
        }
    } else {
        stage_rays_role(g, lane, rb0, nrb, rays_smem, ray_full, ray_empty, flag);
    }
    __syncthreads();
    if (*flag != 0 && threadIdx.x == 0) *static_cast<volatile int*>(g.err) = 1;
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_free(tmem, 2 * kFN);
    }
}

// ---- the same product on CTA pairs (tcgen05 cta_group::2) ---------------------
//
// A cluster of two CTAs computes a 256 x 256 accumulator tile (256 z rows, 128
// x points) with one pair MMA per K step, issued by the even CTA: each CTA
// holds its 128 A rows and half of B (64 x points: their real parts in local
// rows 0..63, their imaginary parts in 64..127), and each keeps its 128
// accumulator rows in its own TMEM. Per 32-ray block a CTA therefore computes
// 128 A and 64 B phasors per ray instead of 128 + 128, stores 64 KB of tiles
// instead of 96 KB, and its tensor core reads half of B from each CTA. The
// accumulator column of x point ix is n = 128 h + 64 c + ix % 64 with
// h = (ix % 128) / 64 (the CTA that holds it) and c = 0 (real), 1 (imaginary).
constexpr int kPStages = 3;
constexpr uint32_t kPA = 128 * 128;              // one A tile (hi or lo): 128 rows x 128 B
constexpr uint32_t kPB = 128 * 128;              // this CTA's half of one B tile
constexpr uint32_t kPStage = 2 * kPA + 2 * kPB;  // A_hi | A_lo | B_hi | B_lo
constexpr int kPProdThreads = 384;               // warps 5..16
constexpr int kPThreads = 32 + kFEpiThreads + kPProdThreads + 32;
constexpr size_t kPSmem =
    1024 + (size_t)kPStages * kPStage + kFRayBufs * kFRayBytes + kFEpiBytes + 256;
static_assert(kPSmem <= 227 * 1024, "pair kernel shared memory");

// Producer warps of a CTA of the pair. Warps 0..7 (ZZ = false) fill 16-byte
// chunk c0 = w (rays 4 c0 .. 4 c0 + 3) of the A rows l, l + 32 and of the B
// rows of x points l, l + 32 (packed pair-rows (A l, B l), (A l+32, B l+32));
// warps 8..11 (ZZ = true) fill chunks c0, c0 + 1 of the A rows 64 + l, 96 + l
// (pair-row (A 64+l, A 96+l)). Every thread thus makes 8 packed phase
// evaluations per ray block; each store instruction of a warp covers 32
// consecutive rows (no bank conflict). Row z index mt*128 + row, x index
// nt*128 + 64 half + point.
template <bool ZZ>
__device__ __forceinline__ void pair_producer(const FusedArgs& g, int c0, int r, int mt, int nt,
                                              uint32_t half, int nrb, unsigned char* tiles,
                                              uint32_t full_lead, uint64_t* empty,
                                              uint64_t* ray_full, uint64_t* ray_empty,
                                              unsigned char* rays_smem, volatile int* flag) {
    using namespace sm100;
    constexpr int NE = ZZ ? 1 : 2;   // pair-rows per thread
    constexpr int NCH = ZZ ? 2 : 1;  // chunks per thread
    bool vx_ok[NE], vy_ok[NE];
    float2 kh2[NE], khn2[NE], kl2[NE], pp2[NE];
#pragma unroll
    for (int e = 0; e < NE; ++e) {
        // (.x, .y) rows: (A r + 32 e, B r + 32 e) or (A 64 + r, A 96 + r).
        const size_t izx = (size_t)mt * 128 + (ZZ ? 64 + r : r + 32 * e);
        vx_ok[e] = izx < g.nz;
        const double ux = vx_ok[e] ? g.zp[izx] - g.oz : 0.0;
        double uy;
        if (ZZ) {
            const size_t izy = (size_t)mt * 128 + 96 + r;
            vy_ok[e] = izy < g.nz;
            uy = vy_ok[e] ? g.zp[izy] - g.oz : 0.0;
        } else {
            const size_t ix = (size_t)nt * 128 + 64 * half + r + 32 * e;
            vy_ok[e] = ix < g.nx;
            uy = vy_ok[e] ? g.xp[ix] - g.ox : 0.0;
        }
        float hx, lx, hy, ly, fx, fy, unused, h0, l0;
        split_coord(-2.0 * g.a_turns * ux, 0.0, &hx, &lx, &unused);
        split_coord(-2.0 * g.a_turns * uy, 0.0, &hy, &ly, &unused);
        split_coord(ux, g.a_turns, &h0, &l0, &fx);
        split_coord(uy, g.a_turns, &h0, &l0, &fy);
        kh2[e] = make_float2(hx, hy);
        khn2[e] = make_float2(-hx, -hy);
        kl2[e] = make_float2(lx, ly);
        pp2[e] = make_float2(fx, fy);
    }
    for (int i = 0; i < nrb; ++i) {
        const int s = i % kPStages, rb = i % kFRayBufs;
        bool ok = mbar_wait(&ray_full[rb], (uint32_t)(i / kFRayBufs) & 1u, g.wait_limit);
        ok = ok && mbar_wait(&empty[s], ((uint32_t)(i / kPStages) & 1u) ^ 1u, g.wait_limit);
        if (!__all_sync(0xffffffffu, ok)) {
            *flag = 1;
            return;
        }
        unsigned char* base = tiles + (size_t)s * kPStage;
        unsigned char* bhi = base + 2 * kPA;
        unsigned char* blo = bhi + kPB;
        const float4* sr = reinterpret_cast<const float4*>(rays_smem + rb * kFRayBytes);
#pragma unroll
        for (int ch = 0; ch < NCH; ++ch) {
            const int c = c0 + ch;
            // [row][ray]: A rows of .x and (ZZ) of .y; B points of .y.
            uint32_t ah[2][4], al[2][4], bh[2][4], bl[2][4];
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
                const int j = 4 * c + jj;
                const float4 v0 = sr[2 * j], v1 = sr[2 * j + 1];
                const float2 rh = ZZ ? f2(v0.x) : make_float2(v0.x, v0.y);
                const float2 rl = ZZ ? f2(v0.z) : make_float2(v0.z, v0.w);
                const float2 rf = ZZ ? f2(v1.x) : make_float2(v1.x, v1.y);
#pragma unroll
                for (int e = 0; e < NE; ++e) {
                    const float2 t = pair_turns2(kh2[e], khn2[e], kl2[e], __fadd2_rn(pp2[e], rf), rh, rl);
                    const float2 th = __fmul2_rn(t, f2(6.28318530717958647692f));
                    float sx, cx, sy, cy;
                    __sincosf(th.x, &sx, &cx);
                    __sincosf(th.y, &sy, &cy);
                    if (!vx_ok[e]) cx = sx = 0.f;
                    split16x2(cx, sx, &ah[ZZ ? 0 : e][jj], &al[ZZ ? 0 : e][jj]);
                    if (ZZ) {
                        if (!vy_ok[e]) cy = sy = 0.f;
                        split16x2(cy, sy, &ah[1][jj], &al[1][jj]);
                    } else {
                        float wr = 0.f, wi = 0.f;
                        if (vy_ok[e]) {
                            wr = cmul_re(v1.z, v1.w, cy, sy);
                            wi = cmul_im(v1.z, v1.w, cy, sy);
                        }
                        split16x2(wr, wi, &bh[e][jj], &bl[e][jj]);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const uint32_t row = (uint32_t)(ZZ ? 64 + r + 32 * k : r + 32 * k);
                *reinterpret_cast<uint4*>(base + sw128(row, c)) =
                    make_uint4(ah[k][0], ah[k][1], ah[k][2], ah[k][3]);
                *reinterpret_cast<uint4*>(base + kPA + sw128(row, c)) =
                    make_uint4(al[k][0], al[k][1], al[k][2], al[k][3]);
            }
            if (!ZZ) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    // Point r + 32 k: (Re W, -Im W) in row r + 32 k, (Im W,
                    // Re W) in row 64 + r + 32 k.
                    const uint32_t row = (uint32_t)(r + 32 * k);
                    *reinterpret_cast<uint4*>(bhi + sw128(row, c)) = make_uint4(
                        neg_hi(bh[k][0]), neg_hi(bh[k][1]), neg_hi(bh[k][2]), neg_hi(bh[k][3]));
                    *reinterpret_cast<uint4*>(bhi + sw128(64 + row, c)) =
                        make_uint4(swap_halves(bh[k][0]), swap_halves(bh[k][1]),
                                   swap_halves(bh[k][2]), swap_halves(bh[k][3]));
                    *reinterpret_cast<uint4*>(blo + sw128(row, c)) = make_uint4(
                        neg_hi(bl[k][0]), neg_hi(bl[k][1]), neg_hi(bl[k][2]), neg_hi(bl[k][3]));
                    *reinterpret_cast<uint4*>(blo + sw128(64 + row, c)) =
                        make_uint4(swap_halves(bl[k][0]), swap_halves(bl[k][1]),
                                   swap_halves(bl[k][2]), swap_halves(bl[k][3]));
                }
            }
        }
        // Make the generic-proxy stores visible to the tensor cores, then one
        // arrival per warp on the even CTA's stage barrier.
        fence_proxy_async();
        __syncwarp();
        if (r == 0) {
            mbar_arrive_cluster(full_lead + 8u * (uint32_t)s);
            mbar_arrive(&ray_empty[rb]);
        }
    }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPThreads, 1)
    fresnel_pair_kernel(FusedArgs g) {
    using namespace sm100;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(tiles + kPStages * kPStage);
    uint64_t* empty = full + kPStages;
    uint64_t* acc_full = empty + kPStages;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* ray_full = acc_empty + 2;
    uint64_t* ray_empty = ray_full + kFRayBufs;
    uint64_t* mma_done = ray_empty + kFRayBufs;  // every issued MMA has completed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
    volatile int* flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    unsigned char* rays_smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(tmem_slot) + 64 + 15) & ~static_cast<uintptr_t>(15));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int mt = blockIdx.x, nt = blockIdx.y, sp = blockIdx.z;
    const uint32_t half = cluster_ctarank(), peer = half ^ 1u;
    const bool leader = half == 0;
    const int rb0 = (int)((long long)g.ray_blocks * sp / g.splits);
    const int rb1 = (int)((long long)g.ray_blocks * (sp + 1) / g.splits);
    const int nrb = rb1 - rb0;
    const int nseg = (nrb + kFSeg - 1) / kFSeg;

    if (threadIdx.x == 0) {
        // full and acc_empty are used in the even CTA only: they collect the
        // arrivals of both CTAs' producer and epilogue warps.
        for (int s = 0; s < kPStages; ++s) {
            mbar_init(&full[s], 2 * kPProdThreads / 32 + (s == 0 ? g.stall : 0u));
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 2 * kFEpiThreads);
        }
        for (int b = 0; b < kFRayBufs; ++b) {
            mbar_init(&ray_full[b], 1);
            mbar_init(&ray_empty[b], kPProdThreads / 32);
        }
        mbar_init(mma_done, 1);
        mbar_init_fence();
        *flag = 0;
    }
    if (warp == 0) tmem_alloc_pair(tmem_slot, 2 * kFN);
    tc_fence_before();
    cluster_sync();  // both CTAs' barriers initialised, TMEM allocated in both
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (leader && lane == 0) {
            // Pair MMA issuer: per ray block three K blocks (hi.hi, hi.lo,
            // lo.hi) of four 256x256x16 steps; segment q accumulates into
            // buffer q & 1 of both CTAs' TMEM.
            constexpr uint32_t idesc = idesc_f16_f32(256, kFN);
            bool good = true;
            for (int q = 0; q < nseg && good; ++q) {
                const int b = q & 1, use = q >> 1;
                if (use >= 1 &&
                    !mbar_wait_cluster(&acc_empty[b], (uint32_t)(use - 1) & 1u, g.wait_limit)) {
                    *flag = 1;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem + (uint32_t)(b * kFN);
                const int i0 = q * kFSeg, i1 = min(nrb, i0 + kFSeg);
                for (int i = i0; i < i1; ++i) {
                    const int s = i % kPStages;
                    if (!mbar_wait_cluster(&full[s], (uint32_t)(i / kPStages) & 1u, g.wait_limit)) {
                        *flag = 1;
                        good = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a_hi = smem_u32(tiles + (size_t)s * kPStage);
                    const uint32_t a_lo = a_hi + kPA, b_hi = a_hi + 2 * kPA, b_lo = b_hi + kPB;
                    const uint32_t as[3] = {a_hi, a_hi, a_lo}, bs[3] = {b_hi, b_lo, b_hi};
#pragma unroll
                    for (int p = 0; p < 3; ++p)
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_f16_pair(d, desc_kmajor_sw128(as[p] + 32u * k),
                                          desc_kmajor_sw128(bs[p] + 32u * k), idesc,
                                          (uint32_t)((i - i0) | p | k));
                    umma_commit_pair(smem_u32(&empty[s]));
                    umma_commit_pair(mapa_shared(&empty[s], peer));
                }
                umma_commit_pair(smem_u32(&acc_full[b]));
                umma_commit_pair(mapa_shared(&acc_full[b], peer));
            }
            // A loop that gave up on a wait may leave MMAs in flight: wait
            // (bounded) for them before either CTA frees its accumulators.
            umma_commit_pair(smem_u32(mma_done));
            if (!mbar_wait(mma_done, 0, max(g.wait_limit, kMmaDrainPolls))) *flag = 1;
        }
        __syncwarp();
    } else if (warp <= 4) {
        unsigned char* tb = rays_smem + kFRayBufs * kFRayBytes + (warp - 1) * 32 * kFEpiRow;
        const uint32_t acc_empty_lead = mapa_shared(acc_empty, 0);
        drain_role(g, warp, lane, mt, nt, sp, nseg, tmem, acc_full, tb, flag, [&](int b) {
            mbar_arrive_cluster(acc_empty_lead + 8u * (uint32_t)b);
        });
    } else if (warp < 5 + kPProdThreads / 32) {
        const int w = warp - 5;
        const uint32_t full_lead = mapa_shared(full, 0);
        if (w < 8)
            pair_producer<false>(g, w, lane, mt, nt, half, nrb, tiles, full_lead, empty, ray_full,
                                 ray_empty, rays_smem, flag);
        else
            pair_producer<true>(g, 2 * (w - 8), lane, mt, nt, half, nrb, tiles, full_lead, empty,
                                ray_full, ray_empty, rays_smem, flag);
    } else {
        stage_rays_role(g, lane, rb0, nrb, rays_smem, ray_full, ray_empty, flag);
    }
    __syncthreads();
    if (*flag != 0 && threadIdx.x == 0) *static_cast<volatile int*>(g.err) = 1;
    tc_fence_before();
    cluster_sync();  // the pair MMAs and all cross-CTA arrivals are done
    if (warp == 0) {
        tc_fence_after();
        tmem_free_pair(tmem, 2 * kFN);
    }
}

// ---- CTA pairs on 256 x points --------------------------------------------------
//
// The wide form of the pair product, 256 z rows x 256 x points per cluster. A row
// of either operand holds a block's 32 real parts, then its 32 imaginary parts, so
// that one B row per x point serves both parts of the field (Re Z Re W - Im Z Im W
// and Re Z Im W + Im Z Re W, the sign a bit of the instruction): half the stores
// per point, and the A phasors serve twice the points. TMEM holds one accumulator
// of 256 columns for the real and one for the imaginary part; a part is drained
// while the other's products run. 2^20
// rays x 512^2 points: 5.30 ms in the form above, 4.78 in this one, of which 0.5 are
// waits for drains (4.28 with segments of 400 blocks; with four epilogue warps 5.16)
// and 3.6 the tensor cores at the 1.55 GHz that the power limit leaves.
constexpr int kWStages = 2;
constexpr uint32_t kWStage = 4 * kPA;  // A_hi | A_lo | B_hi | B_lo, 128 rows each
constexpr int kWEpiWarps = 8;          // warps 1..8, two per quarter of the TMEM lanes
constexpr int kWProdWarps = 8;         // warps 9..16
constexpr int kWThreads = 32 * (1 + kWEpiWarps + kWProdWarps + 1);
constexpr int kWEpiBufs = 4;           // staging buffers per epilogue warp
constexpr uint32_t kWDrainBytes = 32 * 8 * 8;  // 32 rows x 8 columns of the partial
constexpr size_t kWSmem = 1024 + (size_t)kWStages * kWStage + kFRayBufs * kFRayBytes +
                          kWEpiWarps * kWEpiBufs * kWDrainBytes + 256;
static_assert(kWSmem <= 227 * 1024, "wide pair kernel shared memory");

// Element (row, column) of the partials, stored in contiguous blocks of 32 rows x
// 8 columns: one bulk operation drains a block. The 16-byte words of a block's row
// are permuted by the row (conflict-free staging writes).
__device__ __forceinline__ size_t wide_at(size_t row, size_t col, int n_pad) {
    const size_t r = row & 31, c = (col & 7) ^ (((r >> 1) & 3) << 1);
    return ((row >> 5) * (size_t)(n_pad >> 3) + (col >> 3)) * 256 + r * 8 + c;
}

// Producer warp w: rays 8 (w % 4) .. + 7 of the block for the z rows and x points
// 64 (w / 4) .. + 63 (a row and a point of the same number in packed instructions).
// Lanes r and r + 8 hold the same pair and four rays each, so that 16 lanes' 8-byte
// stores cover eight rows' 16-byte words (no bank conflicts). Rows and points past
// the screen's edge hold the phasors of its centre: they only reach accumulators
// nobody reads.
__device__ __forceinline__ void wide_producer(const FusedArgs& g, int w, int lane, int mt, int nt,
                                              uint32_t half, int nrb, unsigned char* tiles,
                                              uint32_t full_lead, uint64_t* empty,
                                              uint64_t* ray_full, uint64_t* ray_empty,
                                              unsigned char* rays_smem, volatile int* flag) {
    using namespace sm100;
    constexpr int NE = 2;  // pairs at a time
    const int sub = (lane >> 3) & 1, oct = w & 3;
    const int row0 = 64 * (w >> 2) + (lane & 7) + ((lane & 16) >> 1);  // + 16 e
    float2 kh2[4], khn2[4], kl2[4], pp2[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const size_t iz = (size_t)mt * 128 + row0 + 16 * e;
        const size_t ix = (size_t)nt * 256 + 128 * half + row0 + 16 * e;
        const double uz = iz < g.nz ? g.zp[iz] - g.oz : 0.0;
        const double ux = ix < g.nx ? g.xp[ix] - g.ox : 0.0;
        float hz, lz, hx, lx, fz, fx, unused, h0, l0;
        split_coord(-2.0 * g.a_turns * uz, 0.0, &hz, &lz, &unused);
        split_coord(-2.0 * g.a_turns * ux, 0.0, &hx, &lx, &unused);
        split_coord(uz, g.a_turns, &h0, &l0, &fz);
        split_coord(ux, g.a_turns, &h0, &l0, &fx);
        kh2[e] = make_float2(hz, hx);
        khn2[e] = make_float2(-hz, -hx);
        kl2[e] = make_float2(lz, lx);
        pp2[e] = make_float2(fz, fx);
    }
    // This thread's 8 bytes of the real and the imaginary 16-byte word of row 0.
    const uint32_t at_re = sw128(row0, oct) + 8 * sub, at_im = sw128(row0, 4 + oct) + 8 * sub;
    for (int i = 0; i < nrb; ++i) {
        const int s = i % kWStages, rb = i % kFRayBufs;
        bool ok = mbar_wait(&ray_full[rb], (uint32_t)(i / kFRayBufs) & 1u, g.wait_limit);
        ok = ok && mbar_wait(&empty[s], ((uint32_t)(i / kWStages) & 1u) ^ 1u, g.wait_limit);
        if (!__all_sync(0xffffffffu, ok)) {
            *flag = 1;
            return;
        }
        unsigned char* base = tiles + (size_t)s * kWStage;
        const float4* sr =
            reinterpret_cast<const float4*>(rays_smem + rb * kFRayBytes) + 2 * (8 * oct + 4 * sub);
#pragma unroll
        for (int e0 = 0; e0 < 4; e0 += NE) {
            uint32_t ah[NE][4], al[NE][4], bh[NE][4], bl[NE][4];  // re, re, im, im
#pragma unroll
            for (int pr = 0; pr < 2; ++pr) {
                float cz[NE][2], sz[NE][2], wr[NE][2], wi[NE][2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float4 v0 = sr[2 * (2 * pr + u)], v1 = sr[2 * (2 * pr + u) + 1];
#pragma unroll
                    for (int e = 0; e < NE; ++e) {
                        const float2 t = pair_turns2(
                            kh2[e0 + e], khn2[e0 + e], kl2[e0 + e],
                            __fadd2_rn(pp2[e0 + e], make_float2(v1.x, v1.y)),
                            make_float2(v0.x, v0.y), make_float2(v0.z, v0.w));
                        const float2 th = __fmul2_rn(t, f2(6.28318530717958647692f));
                        float sx, cx;
                        __sincosf(th.x, &sz[e][u], &cz[e][u]);
                        __sincosf(th.y, &sx, &cx);
                        wr[e][u] = cmul_re(v1.z, v1.w, cx, sx);
                        wi[e][u] = cmul_im(v1.z, v1.w, cx, sx);
                    }
                }
#pragma unroll
                for (int e = 0; e < NE; ++e) {
                    split16x2(cz[e][0], cz[e][1], &ah[e][pr], &al[e][pr]);
                    split16x2(sz[e][0], sz[e][1], &ah[e][2 + pr], &al[e][2 + pr]);
                    split16x2(wr[e][0], wr[e][1], &bh[e][pr], &bl[e][pr]);
                    split16x2(wi[e][0], wi[e][1], &bh[e][2 + pr], &bl[e][2 + pr]);
                }
            }
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                auto put = [&](int tile, const uint32_t(&v)[4]) {
                    unsigned char* o = base + tile * kPA + 16 * 128 * (e0 + e);
                    *reinterpret_cast<uint2*>(o + at_re) = make_uint2(v[0], v[1]);
                    *reinterpret_cast<uint2*>(o + at_im) = make_uint2(v[2], v[3]);
                };
                put(0, ah[e]);
                put(1, al[e]);
                put(2, bh[e]);
                put(3, bl[e]);
            }
        }
        // Make the generic-proxy stores visible to the tensor cores, then one
        // arrival per warp on the even CTA's stage barrier.
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
            mbar_arrive_cluster(full_lead + 8u * (uint32_t)s);
            mbar_arrive(&ray_empty[rb]);
        }
    }
}

// The accumulators' segments (0 real, 1 imaginary) are kFSeg blocks, the imaginary
// part's shifted by half a segment.
constexpr int kWShift = kFSeg / 2;

// Epilogue role (warps 1..8) of the wide form: as drain_role, in blocks of 32 rows
// x 8 columns, the accumulators in turn (the imaginary part's segment ends first).
__device__ __forceinline__ void wide_drain(const FusedArgs& g, int warp, int lane, int mt, int nt,
                                           int sp, int nrb, uint32_t tmem, uint64_t* acc_full,
                                           uint32_t acc_empty_lead, unsigned char* stage,
                                           volatile int* flag) {
    using namespace sm100;
    // Blocks per accumulator and warp, doubles per block.
    constexpr int kBlocks = kFN / 8 / (kWEpiWarps / 4), kBlock = 256;
    const int col0 = (warp - 1) / 4 * (kBlocks * 8);
    const int qd = warp & 3;
    double* row = g.partial + (((size_t)sp * (g.m_pad / 32) + (size_t)mt * 4 + qd) * (g.n_pad / 8) +
                               (size_t)nt * 2 * (kFN / 8) + col0 / 8) * kBlock;
    if (nrb == 0) {
        for (int c = lane; c < kBlocks * kBlock; c += 32) row[c] = row[kFN / 8 * kBlock + c] = 0.0;
        return;
    }
    const int drains = (nrb + kFSeg - 1) / kFSeg + 1 + (max(0, nrb - kWShift) + kFSeg - 1) / kFSeg;
    int buf = 0;
    for (int q = 0; q < drains; ++q) {
        const int b = (q & 1) ^ 1, seg = q >> 1;
        const bool ok = mbar_wait(&acc_full[b], (uint32_t)seg & 1u, g.wait_limit);
        if (!__all_sync(0xffffffffu, ok)) {
            *flag = 1;
            break;
        }
        tc_fence_after();
        double* dst = row + b * (kFN / 8) * kBlock;
#pragma unroll 1
        for (int c = 0; c < kBlocks; c += 2) {
            float v[16];
            tmem_ld_16cols(tmem + ((uint32_t)(qd * 32) << 16) +
                               (uint32_t)(b * kFN + col0 + c * 8),
                           v);
            if (c == kBlocks - 2) {  // the accumulator is free again
                tc_fence_before();
                mbar_arrive_cluster(acc_empty_lead + 8u * (uint32_t)b);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (lane == 0) bulk_wait_read_but<kWEpiBufs - 1>();  // the buffer is free again
                __syncwarp();
                unsigned char* sb = stage + buf * kWDrainBytes;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    reinterpret_cast<double2*>(sb + lane * 64)[k ^ ((lane >> 1) & 3)] =
                        make_double2((double)v[8 * h + 2 * k], (double)v[8 * h + 2 * k + 1]);
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    // The previous segment's operation on this block is performed.
                    bulk_wait_but<2 * kBlocks - 1>();
                    double* to = dst + (c + h) * kBlock;
                    if (seg == 0)
                        bulk_s2g(to, smem_u32(sb), kWDrainBytes);
                    else
                        bulk_add_s2g_f64(to, smem_u32(sb), kWDrainBytes);
                    bulk_commit();
                }
                buf = buf + 1 == kWEpiBufs ? 0 : buf + 1;
            }
        }
    }
    bulk_wait_all();
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kWThreads, 1)
    fresnel_wide_kernel(FusedArgs g) {
    using namespace sm100;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char* rays_smem = tiles + kWStages * kWStage;
    unsigned char* epi_smem = rays_smem + kFRayBufs * kFRayBytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(epi_smem + kWEpiWarps * kWEpiBufs * kWDrainBytes);
    uint64_t* empty = full + kWStages;
    uint64_t* acc_full = empty + kWStages;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* ray_full = acc_empty + 2;
    uint64_t* ray_empty = ray_full + kFRayBufs;
    uint64_t* mma_done = ray_empty + kFRayBufs;  // every issued MMA has completed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
    volatile int* flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int mt = blockIdx.x, nt = blockIdx.y, sp = blockIdx.z;
    const uint32_t half = cluster_ctarank(), peer = half ^ 1u;
    const bool leader = half == 0;
    const int rb0 = (int)((long long)g.ray_blocks * sp / g.splits);
    const int rb1 = (int)((long long)g.ray_blocks * (sp + 1) / g.splits);
    const int nrb = rb1 - rb0;

    if (threadIdx.x == 0) {
        // full and acc_empty are used in the even CTA only: they collect the
        // arrivals of both CTAs' producer and epilogue warps.
        for (int s = 0; s < kWStages; ++s) {
            mbar_init(&full[s], 2 * kWProdWarps + (s == 0 ? g.stall : 0u));
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 2 * 32 * kWEpiWarps);
        }
        for (int b = 0; b < kFRayBufs; ++b) {
            mbar_init(&ray_full[b], 1);
            mbar_init(&ray_empty[b], kWProdWarps);
        }
        mbar_init(mma_done, 1);
        mbar_init_fence();
        *flag = 0;
    }
    if (warp == 0) tmem_alloc_pair(tmem_slot, 2 * kFN);
    tc_fence_before();
    cluster_sync();  // both CTAs' barriers initialised, TMEM allocated in both
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (leader && lane == 0) {
            // Pair MMA issuer: per block hi.hi, hi.lo, lo.hi of four 256x256x16
            // steps into either accumulator. An accumulator is issued first in its
            // segment's last block and last in the next one, so that the other's
            // products of both blocks run while it is drained.
            constexpr uint32_t idesc = idesc_f16_f32(256, kFN);
            bool good = true;
            int end0 = min(nrb, kFSeg), end1 = min(nrb, kWShift), q0 = 0, q1 = 0;
            bool new0 = true, new1 = true;
            for (int i = 0; i < nrb && good; ++i) {
                const int s = i % kWStages;
                if (!mbar_wait_cluster(&full[s], (uint32_t)(i / kWStages) & 1u, g.wait_limit)) {
                    *flag = 1;
                    break;
                }
                tc_fence_after();
                const uint32_t t0 = smem_u32(tiles) + (uint32_t)s * kWStage;
                const uint32_t as[3] = {t0, t0, t0 + kPA};
                const uint32_t bs[3] = {t0 + 2 * kPA, t0 + 3 * kPA, t0 + 2 * kPA};
                const int first = (new0 && i > 0) || i + 1 == end1;
                for (int h = first, t = 0; t < 2; ++t, h ^= 1) {
                    const bool fresh = h ? new1 : new0;
                    const int use = h ? q1 : q0;
                    if (fresh && use >= 1 &&
                        !mbar_wait_cluster(&acc_empty[h], (uint32_t)(use - 1) & 1u, g.wait_limit)) {
                        *flag = 1;
                        good = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t d = tmem + (uint32_t)(h * kFN);
#pragma unroll
                    for (int p = 0; p < 3; ++p)
#pragma unroll
                        for (int k = 0; k < 4; ++k)  // k < 2: A's real parts
                            umma_f16_pair(d, desc_kmajor_sw128(as[p] + 32u * k),
                                          desc_kmajor_sw128(bs[p] + 32u * (h ? k ^ 2 : k)),
                                          h == 0 && k >= 2 ? idesc | kNegateB : idesc,
                                          (uint32_t)(!fresh | p | k));
                    const bool last = i + 1 == (h ? end1 : end0);
                    if (last) {
                        umma_commit_pair(smem_u32(&acc_full[h]));
                        umma_commit_pair(mapa_shared(&acc_full[h], peer));
                    }
                    (h ? new1 : new0) = last;
                    (h ? q1 : q0) += last;
                    if (last) (h ? end1 : end0) = min(nrb, i + 1 + kFSeg);
                }
                umma_commit_pair(smem_u32(&empty[s]));
                umma_commit_pair(mapa_shared(&empty[s], peer));
            }
            // A loop that gave up on a wait may leave MMAs in flight: wait
            // (bounded) for them before either CTA frees its accumulators.
            umma_commit_pair(smem_u32(mma_done));
            if (!mbar_wait(mma_done, 0, max(g.wait_limit, kMmaDrainPolls))) *flag = 1;
        }
        __syncwarp();
    } else if (warp <= kWEpiWarps) {
        wide_drain(g, warp, lane, mt, nt, sp, nrb, tmem, acc_full, mapa_shared(acc_empty, 0),
                   epi_smem + (warp - 1) * kWEpiBufs * kWDrainBytes, flag);
    } else if (warp <= kWEpiWarps + kWProdWarps) {
        wide_producer(g, warp - 1 - kWEpiWarps, lane, mt, nt, half, nrb, tiles,
                      mapa_shared(full, 0), empty, ray_full, ray_empty, rays_smem, flag);
    } else {
        stage_rays_role(g, lane, rb0, nrb, rays_smem, ray_full, ray_empty, flag);
    }
    __syncthreads();
    if (*flag != 0 && threadIdx.x == 0) *static_cast<volatile int*>(g.err) = 1;
    tc_fence_before();
    cluster_sync();  // the pair MMAs and all cross-CTA arrivals are done
    if (warp == 0) {
        tc_fence_after();
        tmem_free_pair(tmem, 2 * kFN);
    }
}

// The ray set's bounds the product needs before it starts: max |es_re|,
// |es_im| (the f16 scaling), max |x - ox| and |z - oz| (the cross-term bound),
// and whether every value is finite. The maxima of non-negative doubles are
// taken on their bit patterns, which order like the values; fmax skips NaN,
// which the finiteness flag reports instead. The last block writes the three
// maxima and the flag to pinned host memory.
__global__ void __launch_bounds__(256) ray_bounds_kernel(const double* __restrict__ rx,
                                                         const double* __restrict__ rz,
                                                         const double* __restrict__ er,
                                                         const double* __restrict__ ei, size_t n,
                                                         double ox, double oz,
                                                         unsigned long long* __restrict__ max_bits,
                                                         int* __restrict__ nonfinite,
                                                         unsigned* __restrict__ ticket,
                                                         unsigned long long* __restrict__ host_out) {
    double m[3] = {0.0, 0.0, 0.0};
    bool bad = false;
    for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < n;
         j += (size_t)gridDim.x * blockDim.x) {
        const double x = rx[j], z = rz[j], a = er[j], b = ei[j];
        m[0] = fmax(m[0], fmax(fabs(a), fabs(b)));
        m[1] = fmax(m[1], fabs(x - ox));
        m[2] = fmax(m[2], fabs(z - oz));
        bad = bad || !isfinite(x + z + a + b);
    }
    __shared__ double sm[8][3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double v = m[k];
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) sm[warp][k] = v;
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicExch(nonfinite, 1);
    __syncthreads();
    if (threadIdx.x < 3) {
        double v = sm[0][threadIdx.x];
        for (int w = 1; w < 8; ++w) v = fmax(v, sm[w][threadIdx.x]);
        atomicMax(max_bits + threadIdx.x, (unsigned long long)__double_as_longlong(v));
    }
    if (!last_block(ticket)) return;
    if (threadIdx.x < 3) host_out[threadIdx.x] = __ldcg(max_bits + threadIdx.x);
    if (threadIdx.x == 3) host_out[3] = (unsigned long long)__ldcg(nonfinite);
}

// acc[iz*nx + ix] (+)= scale * sum over splits of C[iz][n(ix, c)], in FP64 and
// split order. `group`: x points per real / imaginary column group of a 128-point
// block (128 for single-CTA tiles, 64 for CTA pairs); 256 in the wide form, whose
// partials are in the order of wide_at.
__global__ void reduce_kernel(const double* __restrict__ partial, int splits, int m_pad, int n_pad,
                              int group, size_t nz, size_t nx, double scale,
                              double* __restrict__ acc_re, double* __restrict__ acc_im, int first) {
    const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (idx >= nz * nx) return;
    const size_t iz = idx / nx, ix = idx - iz * nx;
    const bool wide = group == 256;
    const size_t loc = ix & 127;
    const size_t col = wide ? (ix >> 8) * 512 + (ix & 255)
                            : (ix >> 7) * kFN + 2 * group * (loc / group) + loc % group;
    const size_t im_off = wide ? 256 / 8 * 256 : group;
    double re = 0.0, im = 0.0;
#pragma unroll 8  // loads ahead of the ordered sums (148 splits: 61 -> 44 us after the product)
    for (int s = 0; s < splits; ++s) {
        const size_t r = (size_t)s * m_pad + iz;
        const double* e = partial + (wide ? wide_at(r, col, n_pad) : r * n_pad + col);
        re += e[0];
        im += e[im_off];
    }
    re *= scale;
    im *= scale;
    if (first) {
        acc_re[idx] = re;
        acc_im[idx] = im;
    } else {
        acc_re[idx] += re;
        acc_im[idx] += im;
    }
}

// ---- host --------------------------------------------------------------------

size_t round_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Words of FresnelWorkspace::host: ray bounds (4 x 8 bytes), then the error word.
constexpr int kFresnelErrWord = 16;

unsigned grid_1d(size_t n, unsigned threads) { return (unsigned)((n + threads - 1) / threads); }

}  // namespace

FresnelShape fresnel_shape(size_t n, size_t nx, size_t nz, int num_sms, bool allow_pair) {
    FresnelShape sh;
    // CTA pairs need an even number of 128-row tiles; a screen of at most 128
    // rows keeps single-CTA tiles rather than padding to 256.
    sh.pair = allow_pair && nz > 128;
    sh.m_pad = round_up(std::max<size_t>(nz, 1), sh.pair ? 256 : 128);
    sh.n_pad = round_up(std::max<size_t>(2 * nx, 1), kFN);
    // The wide form where its product is faster by more than its partials, twice
    // the splits of one tile, cost the sum (20 us): 0.9 of the time per padded pair
    // (5.30 and 4.78 ms on 2^20 rays x 512^2 points), from 1e10 pairs on (sums and
    // all, narrow and wide: 82 and 89 us at 20000 x 256^2, 139 and 142 at 60000,
    // 306 and 290 at 200000).
    const size_t wide_pad = round_up(std::max<size_t>(2 * nx, 1), 2 * kFN);
    sh.wide = sh.pair && 0.9 * (double)wide_pad < (double)sh.n_pad &&
              (double)n * (double)sh.m_pad * (double)(wide_pad / 2) >= 1e10;
    if (sh.wide) sh.n_pad = wide_pad;
    sh.ray_blocks = (int)((n + kFRays - 1) / kFRays);
    sh.tiles = (sh.m_pad / 128) * (sh.n_pad / (sh.wide ? 2 * kFN : kFN));
    // K splits: about one CTA per SM over the output tiles, each split at
    // least ten ray blocks (half a segment) long. 30011 rays x 133 x 101 points:
    // product 113 us with 23 splits of 40 blocks, 80 with 46 of 20, 53 with 74;
    // 10^4 rays x 60 x 500: 101, 72 and 42 us.
    size_t splits = sh.tiles >= (size_t)num_sms ? 1 : (size_t)num_sms / sh.tiles;
    splits = std::min(splits, std::max<size_t>(1, (size_t)sh.ray_blocks / kFMinSplit));
    sh.splits = (int)std::max<size_t>(1, splits);
    return sh;
}

Status fresnel_enqueue(const FresnelIn& in, FresnelWorkspace& ws, cudaStream_t stream,
                       int num_sms, int path, FresnelReport* rep) {
    const size_t n = in.n, nx = in.nx, nz = in.nz, m = nx * nz;
    double* xp = ws.coords.as<double>();
    double* zp = xp + std::max<size_t>(nx, 1);
    coords_kernel<<<grid_1d(nx, 256), 256, 0, stream>>>(in.x_min, in.x_max, nx, xp);
    coords_kernel<<<grid_1d(nz, 256), 256, 0, stream>>>(in.z_min, in.z_max, nz, zp);
    XK_CUDA_TRY(cudaGetLastError());
    rep->kernels += 2;
    const double k = in.energy / kChbar * 1e7;
    const double pre = k / (2.0 * in.dist);
    // Origin of the phase split and the bound on its FP32 cross term.
    const double ox = 0.5 * (in.x_min + in.x_max), oz = 0.5 * (in.z_min + in.z_max);
    const double cross = 2.0 * pre * kInv2Pi *
                         std::max(0.5 * std::fabs(in.x_max - in.x_min) * in.max_rx_off,
                                  0.5 * std::fabs(in.z_max - in.z_min) * in.max_rz_off);
    rep->used_path = path;
    // Non-finite inputs take the FP64 sum, which propagates them as
    // fresnel.rs:53-106 does.
    if (path == XK_PATH_SEPARABLE && n &&
        (!in.finite || (in.max_amp != 0.0 && !(cross < 2097152.0))))
        rep->used_path = path = XK_PATH_F64;
    if (path == XK_PATH_F64 || n == 0 || in.max_amp == 0.0) {
        // FP64 direct sum (with no rays or zero amplitudes it writes zeros).
        const size_t nn = (path == XK_PATH_F64) ? n : 0;
        fresnel_f64_kernel<<<grid_1d(m, kF64Threads), kF64Threads, 0, stream>>>(
            in.rx, in.rz, in.er, in.ei, nn, xp, zp, nx, m, pre, in.out_re, in.out_im);
        XK_CUDA_TRY(cudaGetLastError());
        rep->kernels += 1;
        return Status::Ok();
    }
    const FresnelShape sh = fresnel_shape(n, nx, nz, num_sms, ws.allow_pair);
    XK_TRY(ws.partial.ensure((size_t)sh.splits * sh.m_pad * sh.n_pad * sizeof(double)));
    // Set on every call: the attribute belongs to the current device's
    // context, and a process may use several devices.
    if (sh.wide)
        XK_CUDA_TRY(cudaFuncSetAttribute(fresnel_wide_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWSmem));
    else if (sh.pair)
        XK_CUDA_TRY(cudaFuncSetAttribute(fresnel_pair_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPSmem));
    else
        XK_CUDA_TRY(cudaFuncSetAttribute(fresnel_fused_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFSmem));
    int* err = ws.host.as<int>() + kFresnelErrWord;
    *err = 0;
    FusedArgs fa;
    fa.rx = in.rx;
    fa.rz = in.rz;
    fa.er = in.er;
    fa.ei = in.ei;
    fa.n = n;
    fa.ray_blocks = sh.ray_blocks;
    fa.splits = sh.splits;
    fa.xp = xp;
    fa.zp = zp;
    fa.nx = nx;
    fa.nz = nz;
    fa.a_turns = pre * kInv2Pi;
    fa.inv_scale = 1.0 / in.max_amp;
    fa.ox = ox;
    fa.oz = oz;
    fa.partial = ws.partial.as<double>();
    fa.m_pad = (int)sh.m_pad;
    fa.n_pad = (int)sh.n_pad;
    fa.err = err;
    fa.wait_limit = ws.wait_limit;
    fa.stall = ws.stall_once;
    ws.stall_once = 0;  // armed for one execution
    const dim3 grid((unsigned)(sh.m_pad / 128), (unsigned)(sh.tiles / (sh.m_pad / 128)),
                    (unsigned)sh.splits);
    const bool timed = rep->ev_gemm[0] && rep->ev_gemm[1];
    if (timed) XK_CUDA_TRY(cudaEventRecord(rep->ev_gemm[0], stream));
    if (sh.wide)  // grid.x is even: m_pad is a multiple of 256
        fresnel_wide_kernel<<<grid, kWThreads, kWSmem, stream>>>(fa);
    else if (sh.pair)  // grid.x is even: m_pad is a multiple of 256
        fresnel_pair_kernel<<<grid, kPThreads, kPSmem, stream>>>(fa);
    else
        fresnel_fused_kernel<<<grid, kFThreads, kFSmem, stream>>>(fa);
    XK_CUDA_TRY(cudaGetLastError());
    if (timed) XK_CUDA_TRY(cudaEventRecord(rep->ev_gemm[1], stream));
    reduce_kernel<<<grid_1d(m, 256), 256, 0, stream>>>(ws.partial.as<double>(), sh.splits,
                                                        (int)sh.m_pad, (int)sh.n_pad,
                                                        sh.wide ? 256 : (sh.pair ? 64 : 128), nz, nx,
                                                        in.max_amp, in.out_re, in.out_im, 1);
    XK_CUDA_TRY(cudaGetLastError());
    rep->kernels += 2;
    rep->shape = sh;
    rep->err = err;
    return Status::Ok();
}

}  // namespace xk

// ---- C ABI -------------------------------------------------------------------

namespace {

int fr_fail(xk_ctx* ctx, int code, const std::string& msg) {
    if (ctx) ctx->last_error = msg;
    return code;
}

xk::Status fresnel_host(xk_ctx* ctx, const double* rx, const double* rz, const double* er,
                        const double* ei, size_t n, double energy, double dist,
                        const xk_fresnel_screen* sc, double* amp_re, double* amp_im,
                        double* x_pixels, double* z_pixels, int path, xk_stats* stats) {
    cudaStream_t s = ctx->stream;
    ctx->pending.clear();
    xk::FresnelWorkspace& ws = ctx->fresnel;
    const size_t nx = sc->nx, nz = sc->nz, m = nx * nz;
    const size_t nb = n * sizeof(double);
    XK_TRY(ctx->in_rays.ensure(std::max<size_t>(4 * nb, 8)));
    XK_TRY(ws.coords.ensure((std::max<size_t>(nx, 1) + std::max<size_t>(nz, 1)) * sizeof(double)));
    XK_TRY(ctx->out_field.ensure(std::max<size_t>(2 * m * sizeof(double), 8)));
    XK_TRY(ws.host.ensure(256));
    double* d = ctx->in_rays.as<double>();
    const double* src[4] = {rx, rz, er, ei};
    XK_TRY(xk::stage_in(ctx, src, 4, d, n, 0, s));
    double max_amp = 0.0, max_rx = 0.0, max_rz = 0.0;
    const double ox = 0.5 * (sc->x_min + sc->x_max), oz = 0.5 * (sc->z_min + sc->z_max);
    bool finite = true;
    int bounds_kernels = 0;
    if (n) {
        // The bounds come from the uploaded columns on the device (a host
        // loop over 2^20 rays takes milliseconds), which writes them here.
        XK_TRY(ws.ctrl.ensure(256));
        unsigned long long* d_max = ws.ctrl.as<unsigned long long>();
        int* d_bad = reinterpret_cast<int*>(d_max + 3);
        unsigned* ticket = reinterpret_cast<unsigned*>(d_max + 4);
        XK_CUDA_TRY(cudaMemsetAsync(d_max, 0, 5 * sizeof(unsigned long long), s));
        const unsigned blocks =
            (unsigned)std::min<size_t>((n + 255) / 256, (size_t)std::max(ctx->num_sms, 1) * 4);
        unsigned long long* h = ws.host.as<unsigned long long>();
        xk::ray_bounds_kernel<<<blocks, 256, 0, s>>>(d, d + n, d + 2 * n, d + 3 * n, n, ox, oz,
                                                     d_max, d_bad, ticket, h);
        XK_CUDA_TRY(cudaGetLastError());
        bounds_kernels = 1;
        XK_CUDA_TRY(cudaStreamSynchronize(s));
        double v[3];
        std::memcpy(v, h, sizeof(v));
        // An upper bound of |es_j| is all the f16 scaling needs.
        max_amp = v[0];
        max_rx = v[1];
        max_rz = v[2];
        finite = h[3] == 0;
    }
    max_amp *= 1.4142135623730951;
    double* out = ctx->out_field.as<double>();
    xk::FresnelIn in{d, d + n, d + 2 * n, d + 3 * n, n, energy, dist,
                     sc->x_min, sc->x_max, sc->z_min, sc->z_max, nx, nz, max_amp, max_rx, max_rz,
                     out, out + m, finite};
    xk::FresnelReport rep;
    const bool timed = stats && path == XK_PATH_SEPARABLE;
    if (timed) {
        for (auto& e : ws.ev)
            if (!e) XK_CUDA_TRY(cudaEventCreate(&e));
        rep.ev_gemm[0] = ws.ev[0];
        rep.ev_gemm[1] = ws.ev[1];
    }
    XK_CUDA_TRY(cudaEventRecord(ctx->ev0, s));
    xk::Status st = xk::fresnel_enqueue(in, ws, s, ctx->num_sms, path, &rep);
    if (st.ok()) st = xk::Status::FromCuda(cudaEventRecord(ctx->ev1, s));
    double* const fields[2] = {amp_re, amp_im};
    if (st.ok()) st = xk::stage_out(ctx, fields, 2, out, m, 0, s);
    const double* xp = ws.coords.as<double>();
    if (st.ok() && x_pixels && nx) st = xk::stage_out(ctx, &x_pixels, 1, xp, nx, 2 * m, s);
    if (st.ok() && z_pixels && nz)
        st = xk::stage_out(ctx, &z_pixels, 1, xp + std::max<size_t>(nx, 1), nz, 2 * m + nx, s);
    if (st.ok()) st = xk::Status::FromCuda(cudaStreamSynchronize(s));
    XK_TRY(st);
    if (rep.err && *rep.err)
        return xk::Status::Err(XK_ERR_TIMEOUT, "tensor-core product: a bounded wait ran out");
    xk::unstage(ctx);
    if (timed && rep.used_path == XK_PATH_SEPARABLE && rep.err) {
        float ms = 0.f;
        XK_CUDA_TRY(cudaEventElapsedTime(&ms, ws.ev[0], ws.ev[1]));
        rep.gemm_ms = ms;
    }
    if (stats) {
        float ms = 0.f;
        XK_CUDA_TRY(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
        stats->gpu_ms = ms;
        stats->main_kernel_ms = rep.gemm_ms;
        stats->kernels = rep.kernels + bounds_kernels;
        stats->path = rep.used_path;
        stats->pairs = (double)n * (double)m;
        stats->h2d_bytes = 4.0 * nb;
        stats->d2h_bytes = 2.0 * m * sizeof(double) + (double)(nx + nz) * sizeof(double);
        stats->n_chunks = rep.shape.ray_blocks;
        stats->n_tiles = (int)rep.shape.tiles;
        stats->groups = rep.shape.splits;
        stats->n_items = (long long)rep.shape.tiles * rep.shape.splits;
        stats->sweep = rep.used_path == XK_PATH_SEPARABLE ? (rep.shape.pair ? 1 : 0) : -1;
    }
    return xk::Status::Ok();
}

}  // namespace

extern "C" int xk_fresnel_propagate(xk_ctx* ctx, const double* ray_x, const double* ray_z,
                                    const double* es_re, const double* es_im, size_t n_rays,
                                    double energy, double dist, const xk_fresnel_screen* screen,
                                    double* amp_re, double* amp_im, double* x_pixels,
                                    double* z_pixels, int path, xk_stats* stats) {
    if (!ctx) return XK_ERR_INVALID;
    if (!screen) return fr_fail(ctx, XK_ERR_INVALID, "null screen");
    if (path != XK_PATH_F64 && path != XK_PATH_SEPARABLE)
        return fr_fail(ctx, XK_ERR_INVALID, "unknown path (F64 or SEPARABLE)");
    const size_t nx = screen->nx, nz = screen->nz;
    if (nx && nz > SIZE_MAX / nx) return fr_fail(ctx, XK_ERR_INVALID, "nx * nz overflows");
    if (nx > (size_t)1 << 30 || nz > (size_t)1 << 30)
        return fr_fail(ctx, XK_ERR_INVALID, "screen too large");
    auto t0 = std::chrono::steady_clock::now();
    if (stats) std::memset(stats, 0, sizeof(*stats));
    if (nx * nz == 0) return XK_OK;
    if (n_rays && (!ray_x || !ray_z || !es_re || !es_im))
        return fr_fail(ctx, XK_ERR_INVALID, "null ray array");
    if (!amp_re || !amp_im) return fr_fail(ctx, XK_ERR_INVALID, "null output array");
    std::lock_guard<std::mutex> lock(ctx->mu);
    cudaSetDevice(ctx->device);
    xk::Status st = fresnel_host(ctx, ray_x, ray_z, es_re, es_im, n_rays, energy, dist, screen,
                                 amp_re, amp_im, x_pixels, z_pixels, path, stats);
    if (!st.ok()) return fr_fail(ctx, st.code, st.msg);
    if (stats)
        stats->wall_ms =
            std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0)
                .count();
    return XK_OK;
}
