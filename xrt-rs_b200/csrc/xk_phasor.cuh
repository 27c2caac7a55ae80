// Device pieces shared by the tensor-core products (xk_fresnel.cu,
// xk_grid.cu): exact FP32 evaluation of large phases, the f16 hi + lo split,
// the swizzled tile layout and the accumulator drains.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

#include "xk_sm100.cuh"

namespace xk {
namespace phasor {

constexpr int kFRays = 32;         // rays per block: K = 64 halves (re, im)
constexpr int kFEpiThreads = 128;  // warps 1..4
constexpr int kFRayBufs = 4;       // staged ray blocks in flight
constexpr int kFSeg = 20;          // ray blocks per f32 segment (xk_fresnel.cu)
// Polls of the issuer's final wait for its MMAs (never fewer, whatever the
// caller's wait limit): the accumulators are freed after it.
constexpr uint32_t kMmaDrainPolls = 1u << 22;
constexpr int kFN = 256;                         // accumulator columns (N of the UMMA)
// Epilogue staging: per epilogue warp 32 rows of 16 FP64 values, rows 144
// bytes apart (16-byte stores of 32 lanes then meet all banks once).
constexpr uint32_t kFEpiRow = 144;
constexpr uint32_t kFEpiBytes = 4 * 32 * kFEpiRow;
// Byte offset of 16-byte chunk c (0..7) of row r in a 128-byte-swizzled tile.
__device__ __forceinline__ uint32_t sw128(uint32_t r, uint32_t c) {
    return r * 128u + ((c ^ (r & 7u)) << 4);
}

// Phase split. With p, r relative to the screen centre the phase in turns is
//     t = a (p - r)^2 = P(p) + kappa(p) r + R(r),
//     P = frac(a p^2), R = frac(a r^2), kappa = -2 a p,
// where P and R are reduced in FP64 once per screen row and per ray. The
// cross term kappa r (up to 2^21 turns, checked on the host) is formed
// exactly in FP32 from hi/lo splits of kappa and r: the rounded product
// kh*rh, its FMA error term, and the two small cross products; its integer
// part drops out and the fractional remainder keeps ~1e-7 turn.
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: (x + kMagic) - kMagic = rint(x), |x| < 2^22

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }

// The same for a row of A (.x) and a row of B (.y) at once on sm_100's packed
// f32x2 instructions, with the operation sequence and roundings of the scalar
// form: p1 = kh rh rounded, e1 = its FMA error, f1 = p1 - rint(p1),
// t = (pr + f1) + (kh rl + kl rh + e1), result t - rint(t). rint is the
// magic-number rounding (exact and sign-symmetric for |x| < 2^22), and the
// product is carried negated (khn = -kh) so that every step is one packed
// FMA, multiply or add; a - b is formed as fma(b, -1, a).
__device__ __forceinline__ float2 pair_turns2(float2 kh, float2 khn, float2 kl, float2 pr,
                                              float2 rh, float2 rl) {
    const float2 m = f2(kMagic), mn = f2(-kMagic), one_n = f2(-1.f);
    const float2 p1n = __fmul2_rn(khn, rh);                          // -p1
    const float2 e1 = __ffma2_rn(kh, rh, p1n);                       // kh rh - p1
    const float2 r1 = __fadd2_rn(__fadd2_rn(p1n, m), mn);            // rint(-p1)
    const float2 f1n = __ffma2_rn(r1, one_n, p1n);                   // -f1
    float2 sm = __ffma2_rn(kh, rl, e1);
    sm = __ffma2_rn(kl, rh, sm);
    const float2 t = __fadd2_rn(__ffma2_rn(f1n, one_n, pr), sm);    // (pr + f1) + sm
    const float2 rt = __fadd2_rn(__fadd2_rn(t, m), mn);
    return __ffma2_rn(rt, one_n, t);                                 // t - rint(t)
}

// hi/lo float split of a double and frac(a v^2) as a float.
__device__ __forceinline__ void split_coord(double v, double a, float* hi, float* lo, float* fr) {
    *hi = (float)v;
    *lo = (float)(v - (double)*hi);
    const double t = (a * v) * v;
    *fr = (float)(t - rint(t));
}

// (a, b) -> f16x2 hi (round to nearest) and f16x2 lo = (a, b) - hi.
__device__ __forceinline__ void split16x2(float a, float b, uint32_t* hi, uint32_t* lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 back = __half22float2(h);
    const float2 d = __ffma2_rn(back, f2(-1.f), make_float2(a, b));
    const __half2 l = __floats2half2_rn(d.x, d.y);
    *hi = *reinterpret_cast<const uint32_t*>(&h);
    *lo = *reinterpret_cast<const uint32_t*>(&l);
}

// (a, b) -> f16x2, rounded to nearest.
__device__ __forceinline__ uint32_t pack16x2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// (a + ib)(c + is) with explicit roundings, so that every kernel variant forms
// the same W bit for bit (no compiler-chosen FMA contraction).
__device__ __forceinline__ float cmul_re(float a, float b, float c, float s) {
    return __fmaf_rn(a, c, __fmul_rn(-b, s));
}
__device__ __forceinline__ float cmul_im(float a, float b, float c, float s) {
    return __fmaf_rn(a, s, __fmul_rn(b, c));
}

// (x, y) -> (x, -y) and (y, x) on packed f16 pairs (sign flip, half swap).
__device__ __forceinline__ uint32_t neg_hi(uint32_t v) { return v ^ 0x80000000u; }
__device__ __forceinline__ uint32_t swap_halves(uint32_t v) { return __byte_perm(v, 0, 0x1032); }

}  // namespace phasor
}  // namespace xk
