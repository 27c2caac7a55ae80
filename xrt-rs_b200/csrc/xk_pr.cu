// FP32 phase-reduced Kirchhoff path.
//
// Phase decomposition. For a screen tile t (centre P0) and a ray chunk c
// (centre R0, all rays of one energy, wavenumber k) write q = p - R0 for a
// screen point p, rho = r - R0 for a ray r, and u = (P0 - R0)/|P0 - R0|.
// Then exactly
//     |p - r| = |q| - u.rho + Delta,
//     Delta   = (|rho_perp|^2 - 2 v.rho) / (|p - r| + |q| - u.rho),
// with v = q - |q| u (|v| <= tile radius) and rho_perp = rho - (u.rho) u.
// The denominator equals 2(|q| - u.rho) + Delta. The kernel uses 2(|q| - u.rho),
// which changes the phase by k Delta^2 / (2|q|): half the tolerance at most, by
// the planner's cap of the residual phase (pair_budget).
//   * exp(i k |q|)      per screen point and chunk: reference path length and
//                       its turn count in FP64, sin/cos of the reduced turn,
//   * exp(-i k u.rho)   per ray and item, FP64 argument reduction folded
//                       into the ray's amplitudes,
//   * exp(i k Delta)    per pair, FP32: |k Delta| <= the residual-phase
//                       budget by construction of the chunk grid (the budget
//                       follows from the requested tolerance).
// This generalises the reference's single-centroid reduction
// (src/gpu/shaders/kirchhoff.wgsl:95-113, src/gpu/kirchhoff.rs:96-104,
// 276-297), whose FP32 residual is unbounded at high Fresnel numbers.
//
// Work decomposition. Screen points are sorted along a Hilbert curve and cut
// into tiles of 32*kPrPpl points (one warp, kPrPpl points per lane). Rays are
// binned into a grid of cells sized so that the residual phase bound holds
// for every (tile, cell) pair; each occupied cell is a chunk. The sorted ray
// list is cut into `groups` equal ranges; an item is (tile, range), and the
// persistent kernel's warps claim items from an atomic counter. Inside an
// item the range is streamed through shared memory kPrStage rays at a time by
// cp.async.bulk (TMA bulk copy, mbarrier completion, two buffers), prepared
// in place for the item's direction u, and swept by all 32 lanes. Each lane
// keeps per-point FP32 partial sums folded every stage into two-float
// (TwoSum) accumulators; at a chunk boundary they are multiplied by the
// per-point phasor and added, in FP64, to the item's slot. A final pass adds
// the `groups` slots of every point in order, so results are deterministic.
//
// Two sweeps: the SFU sweep (rcp.approx for 1/(2|q| - 2u.rho)) and the packed
// sweep, which processes two screen points per instruction with the sm_100
// f32x2 FMA and replaces the reciprocal by the series
// r0 (1 + e + e^2), r0 = 1/(2|q|), e = 2u.rho r0, when the planner can bound
// |e| (the neglected e^3 term then stays below 1e-8 relative).

#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "xk_dd.cuh"
#include "xk_pr.cuh"
#include "xk_sm100.cuh"

namespace xk {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kSumFields = 41;
// |e| bound under which the packed sweep's series reciprocal is used.
constexpr double kSeriesRcpBound = 2e-3;
// Fold the base phase when the estimated chunks per ray group reach this.
constexpr double kFoldChunksPerGroup = 4.0;
// ... and chunks average fewer rays than this: a chunk switch (the points'
// double-double base phase and the flush of the chunk sums) costs about as
// much as sweeping 30 rays, the folded sweep about 8 % more per ray.
constexpr double kFoldRaysPerChunk = 512.0;
// Largest |es_j ep_0 - ep_j es_0| / (|es_j| |ep_0| + |ep_j| |es_0|) over the
// rays under which every ray counts as having ray 0's polarization (2^-24:
// the per-ray deviation is then below the FP32 rounding of the amplitudes
// that the kernel applies anyway).
constexpr double kOnePolTol = 5.9604644775390625e-8;
// Amplitude components the phase-reduced kernels carry in FP32: their partial
// sums over a chunk (up to 2^20 rays, |U| up to ~1/path) must stay inside
// FP32's range, and products with |U| must stay normal.
constexpr double kF32AmpMax = 1e30, kF32AmpMin = 1e-30;

// ---------------------------------------------------------------------------
// Planner kernels
// ---------------------------------------------------------------------------

enum : int { OP_SUM = 0, OP_MIN = 1, OP_MAX = 2 };
// How field i of a solve's summary combines.
__host__ __device__ constexpr int sum_op(int i) {
    switch (i) {
        case 3: case 4: case 5:        // ray bbox
        case 9:                        // energy range
        case 11: case 12: case 13:     // normal range
        case 20: case 21: case 22:     // screen bbox
        case 33:                       // inner length of a rectangular screen
        case 34:                       // nl range
            return OP_MIN;
        case 6: case 7: case 8:
        case 10:
        case 14: case 15: case 16:
        case 23: case 24: case 25:
        case 27:                       // polarization deviation
        case 32: case 40:              // largest component of es, of ep
        case 35:
            return OP_MAX;
        default:  // 0-2 ray and 17-19 screen position sums, 26 non-finite probe, 28-31
                  // ray 0's es and ep, 36 squared distances from ray 0, 37-39 its position
            return OP_SUM;
    }
}

__device__ __forceinline__ double op_combine(int op, double a, double b) {
    return op == OP_SUM ? a + b : (op == OP_MIN ? fmin(a, b) : fmax(a, b));
}

// One partial summary per block over rays and screen points. The last field
// sums every input value times zero: 0 when all are finite, NaN otherwise
// (fmin / fmax skip NaN, so the boxes alone would not show it). Fields 27-31
// test whether all rays share ray 0's polarization: the largest relative
// |es_j ep_0 - ep_j es_0|, and ray 0's (es, ep); fields 32 and 40 are the largest
// components of es and of ep. Field 33 is the first point at which a coordinate that
// points 0 and 1 share changes: the inner length if the screen is rectangular
// (infinite if points 0 and 1 differ in none or several coordinates). Clears
// `probe` for the check of that order. The last block combines the rows into row
// `blocks` and into pinned host memory, which the host reads after its next
// synchronisation (a copy of a few hundred bytes costs more than the kernel).
// A launch serves up to N solves: one of a batch's solves fills few SMs and takes
// its latency whatever its size (16 uneven solves: 291 us one after another, 60 in
// one launch).
struct SummaryArgs {
    RaysDev rays;
    PixDev pix;
    int n, m;
    int first, blocks;  // of the grid's blocks
    double* block_out;
    GridProbe* probe;
    unsigned* ticket;
    double* host_out;
};
template <int N>
struct SummaryBatch {
    SummaryArgs s[N];
};

template <int N>
__global__ void __launch_bounds__(256)
    summary_kernel(const __grid_constant__ SummaryBatch<N> batch) {
    const SummaryArgs& A = solve_of_block(batch.s);
    const RaysDev& r = A.rays;
    const PixDev& p = A.pix;
    const int n = A.n, m = A.m, block = (int)blockIdx.x - A.first;
    double* const block_out = A.block_out;
    if (block == 0 && threadIdx.x == 0) *A.probe = GridProbe{};
    // Fields 32 and 40 as floats, rounded up: as doubles they cost the registers of the
    // second block per SM (2^18 rays x 256^2 points: 33 us so, 40 as doubles, 30.5 with
    // one double for both).
    float amp[2] = {0.f, 0.f};
    double f[kSumFields];
#pragma unroll
    for (int i = 0; i < kSumFields; ++i)
        f[i] = sum_op(i) == OP_SUM ? 0.0 : (sum_op(i) == OP_MIN ? INFINITY : -INFINITY);
    const int stride = A.blocks * 256;
    const double a0r = r.es_re[0], a0i = r.es_im[0], b0r = r.ep_re[0], b0i = r.ep_im[0];
    const double a0n = sqrt(a0r * a0r + a0i * a0i), b0n = sqrt(b0r * b0r + b0i * b0i);
    const double x0 = r.x[0], y0 = r.y[0], z0 = r.z[0];
    const double q0 = p.x[0], q1 = p.y[0], q2 = p.z[0];
    const int one = m > 1 ? 1 : 0;
    const bool in0 = p.x[one] != q0, in1 = p.y[one] != q1, in2 = p.z[one] != q2;
    const bool ordered = (int)in0 + (int)in1 + (int)in2 == 1;
    for (int i = block * 256 + threadIdx.x; i < n; i += stride) {
        double x = r.x[i], y = r.y[i], z = r.z[i], e = r.energy[i];
        double a = r.nx[i], b = r.ny[i], c = r.nz[i];
        f[0] += x; f[1] += y; f[2] += z;
        f[3] = fmin(f[3], x); f[4] = fmin(f[4], y); f[5] = fmin(f[5], z);
        f[6] = fmax(f[6], x); f[7] = fmax(f[7], y); f[8] = fmax(f[8], z);
        f[9] = fmin(f[9], e); f[10] = fmax(f[10], e);
        f[11] = fmin(f[11], a); f[12] = fmin(f[12], b); f[13] = fmin(f[13], c);
        f[14] = fmax(f[14], a); f[15] = fmax(f[15], b); f[16] = fmax(f[16], c);
        const double ar = r.es_re[i], ai = r.es_im[i], br = r.ep_re[i], bi = r.ep_im[i];
        const double nl = r.nl[i];
        f[34] = fmin(f[34], nl);
        f[35] = fmax(f[35], nl);
        const double ux = x - x0, uy = y - y0, uz = z - z0;
        f[36] += ux * ux + uy * uy + uz * uz;
        f[26] += (x + y + z + e + a + b + c + nl + ar + ai + br + bi) * 0.0;
        const double dr = (ar * b0r - ai * b0i) - (br * a0r - bi * a0i);
        const double di = (ar * b0i + ai * b0r) - (br * a0i + bi * a0r);
        const double nrm = sqrt(ar * ar + ai * ai) * b0n + sqrt(br * br + bi * bi) * a0n;
        const double dn = sqrt(dr * dr + di * di);
        f[27] = fmax(f[27], nrm > 0.0 ? dn / nrm : (dn > 0.0 ? INFINITY : 0.0));
        amp[0] = fmaxf(amp[0], __double2float_ru(fmax(fabs(ar), fabs(ai))));
        amp[1] = fmaxf(amp[1], __double2float_ru(fmax(fabs(br), fabs(bi))));
        if (i == 0) {
            f[28] += ar;
            f[29] += ai;
            f[30] += br;
            f[31] += bi;
            f[37] += x;
            f[38] += y;
            f[39] += z;
        }
    }
    for (int i = block * 256 + threadIdx.x; i < m; i += stride) {
        double x = p.x[i], y = p.y[i], z = p.z[i];
        f[17] += x; f[18] += y; f[19] += z;
        f[20] = fmin(f[20], x); f[21] = fmin(f[21], y); f[22] = fmin(f[22], z);
        f[23] = fmax(f[23], x); f[24] = fmax(f[24], y); f[25] = fmax(f[25], z);
        f[26] += (x + y + z) * 0.0;
        if (ordered && ((!in0 && x != q0) || (!in1 && y != q1) || (!in2 && z != q2)))
            f[33] = fmin(f[33], (double)i);
    }
    __shared__ double sm[8][kSumFields];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < kSumFields; ++i) {
        if (i == 32 || i == 40) {
            float v = amp[i == 40];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o));
            if (lane == 0) sm[warp][i] = v;
            continue;
        }
        double v = f[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = op_combine(sum_op(i), v, __shfl_xor_sync(kFull, v, o));
        if (lane == 0) sm[warp][i] = v;
    }
    __syncthreads();
    if (threadIdx.x < kSumFields) {
        int i = threadIdx.x;
        double v = sm[0][i];
        const int op = sum_op(i);
        for (int w = 1; w < 8; ++w) v = op_combine(op, v, sm[w][i]);
        block_out[block * kSumFields + i] = v;
    }
    if (!last_block(A.ticket, A.blocks)) return;
    constexpr int kParts = 6;  // threads per field
    __shared__ double sp[kParts][kSumFields];
    const int rows = A.blocks, i = threadIdx.x % kSumFields, part = threadIdx.x / kSumFields;
    const int op = sum_op(i);
    if (part < kParts) {
        double v = op == OP_SUM ? 0.0 : (op == OP_MIN ? INFINITY : -INFINITY);
#pragma unroll 4
        for (int b = part; b < rows; b += kParts)
            v = op_combine(op, v, __ldcg(block_out + b * kSumFields + i));
        sp[part][i] = v;
    }
    __syncthreads();
    if (threadIdx.x < kSumFields) {
        double v = sp[0][i];
        for (int w = 1; w < kParts; ++w) v = op_combine(op, v, sp[w][i]);
        block_out[rows * kSumFields + i] = v;
        A.host_out[i] = v;
    }
}

struct Frame {
    double ox, oy, oz;  // origin
    double e1[3], e2[3], u0[3];
    double lo[3], scale[3];  // quantisation: q_a = (coord_a - lo_a) * scale_a
};

__device__ __forceinline__ void to_frame(const Frame& fr, double x, double y, double z,
                                         double out[3]) {
    double dx = x - fr.ox, dy = y - fr.oy, dz = z - fr.oz;
    out[0] = dx * fr.e1[0] + dy * fr.e1[1] + dz * fr.e1[2];
    out[1] = dx * fr.e2[0] + dy * fr.e2[1] + dz * fr.e2[2];
    out[2] = dx * fr.u0[0] + dy * fr.u0[1] + dz * fr.u0[2];
}

__device__ __forceinline__ uint32_t quant(double v, double maxv) {
    double q = floor(v);
    q = fmin(fmax(q, 0.0), maxv);
    return (uint32_t)q;
}

// Distance of (x, y) along the Hilbert curve of order 16 (the classic
// iterative xy -> d mapping: quadrant digit per level, then rotate/flip).
__device__ __forceinline__ uint32_t hilbert16(uint32_t x, uint32_t y) {
    uint32_t d = 0;
    for (uint32_t s = 1u << 15; s > 0; s >>= 1) {
        uint32_t rx = (x & s) ? 1u : 0u;
        uint32_t ry = (y & s) ? 1u : 0u;
        d += s * s * ((3u * rx) ^ ry);
        if (ry == 0) {
            if (rx == 1) {
                x = 0xffffu - x;
                y = 0xffffu - y;
            }
            uint32_t t = x;
            x = y;
            y = t;
        }
    }
    return d;
}

// Hilbert key of every screen point over its two transverse frame axes, the
// longitudinal coordinate as tie-break.
// Clears the tile extents for the next kernel.
__global__ void pixel_keys_kernel(PixDev p, int m, Frame fr, uint64_t* __restrict__ keys,
                                  int* __restrict__ idx,
                                  unsigned long long* __restrict__ amax_bits) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 4) amax_bits[i] = 0;
    if (i >= m) return;
    double c[3];
    to_frame(fr, p.x[i], p.y[i], p.z[i], c);
    uint32_t hx = quant((c[0] - fr.lo[0]) * fr.scale[0], 65535.0);
    uint32_t hy = quant((c[1] - fr.lo[1]) * fr.scale[1], 65535.0);
    uint32_t hz = quant((c[2] - fr.lo[2]) * fr.scale[2], 2097151.0);
    keys[i] = ((uint64_t)hilbert16(hx, hy) << 21) | hz;
    idx[i] = i;
}

// One warp per tile: slot table, slot-ordered coordinates, bounding-box
// centre; the largest radius of any tile, its largest extents across and along
// the frame's long axis u0 (amax_bits[0..2]) and the sum of the tiles' extents
// across (amax_bits[3], in units of 1 / sum_scale: an integer, so that it does not
// depend on the order of the tiles), which the last block writes to pinned host memory.
// Centres are snapped to multiples of `quantum` as the chunk centres are, so
// that differences between points, tile and chunk centres are exact. rel, ns:
// each slot's offset from the centre (PrSolve::tile_rel); n2 = 2 n for solves
// of one normal.
__global__ void tile_kernel(PixDev p, int m, int n_tiles, Frame fr, double quantum,
                            double inv_quantum, double sum_scale, double3 n2,
                            const int* __restrict__ sorted_idx, double4* __restrict__ rel,
                            float* __restrict__ ns, int* __restrict__ tile_perm, double* __restrict__ tpx,
                            double* __restrict__ tpy, double* __restrict__ tpz,
                            double* __restrict__ tile_center,
                            unsigned long long* __restrict__ amax_bits,
                            unsigned* __restrict__ ticket, double* __restrict__ host_out) {
    int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (t < n_tiles) {
        double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (int i = 0; i < kPrPpl; ++i) {
            long long s = (long long)t * kPrTile + lane + 32 * i;
            int id = s < m ? sorted_idx[s] : -1;
            tile_perm[s] = id;
            if (id >= 0) {
                double v[3] = {p.x[id], p.y[id], p.z[id]};
                for (int a = 0; a < 3; ++a) {
                    lo[a] = fmin(lo[a], v[a]);
                    hi[a] = fmax(hi[a], v[a]);
                }
            }
        }
        for (int a = 0; a < 3; ++a)
            for (int o = 16; o > 0; o >>= 1) {
                lo[a] = fmin(lo[a], __shfl_xor_sync(kFull, lo[a], o));
                hi[a] = fmax(hi[a], __shfl_xor_sync(kFull, hi[a], o));
            }
        double c[3];
        for (int a = 0; a < 3; ++a) c[a] = rint(0.5 * (lo[a] + hi[a]) * inv_quantum) * quantum;
        double rad = 0.0, across = 0.0, along = 0.0;
        for (int i = 0; i < kPrPpl; ++i) {
            long long s = (long long)t * kPrTile + lane + 32 * i;
            int id = s < m ? sorted_idx[s] : -1;
            double x = c[0], y = c[1], z = c[2];
            if (id >= 0) {
                x = p.x[id];
                y = p.y[id];
                z = p.z[id];
                double dx = x - c[0], dy = y - c[1], dz = z - c[2];
                rad = fmax(rad, sqrt(dx * dx + dy * dy + dz * dz));
                const double f1 = dx * fr.e1[0] + dy * fr.e1[1] + dz * fr.e1[2];
                const double f2 = dx * fr.e2[0] + dy * fr.e2[1] + dz * fr.e2[2];
                across = fmax(across, sqrt(f1 * f1 + f2 * f2));
                along = fmax(along, fabs(dx * fr.u0[0] + dy * fr.u0[1] + dz * fr.u0[2]));
            }
            tpx[s] = x;
            tpy[s] = y;
            tpz[s] = z;
            const double sx = x - c[0], sy = y - c[1], sz = z - c[2];
            rel[s] = make_double4(sx, sy, sz, sx * sx + sy * sy + sz * sz);
            ns[s] = (float)(n2.x * sx + n2.y * sy + n2.z * sz);
        }
        for (int o = 16; o > 0; o >>= 1) {
            rad = fmax(rad, __shfl_xor_sync(kFull, rad, o));
            across = fmax(across, __shfl_xor_sync(kFull, across, o));
            along = fmax(along, __shfl_xor_sync(kFull, along, o));
        }
        if (lane == 0) {
            tile_center[3 * t + 0] = c[0];
            tile_center[3 * t + 1] = c[1];
            tile_center[3 * t + 2] = c[2];
            atomicMax(amax_bits, (unsigned long long)__double_as_longlong(rad));
            atomicMax(amax_bits + 1, (unsigned long long)__double_as_longlong(across));
            atomicMax(amax_bits + 2, (unsigned long long)__double_as_longlong(along));
            atomicAdd(amax_bits + 3, (unsigned long long)rint(across * sum_scale));
        }
    }
    if (last_block(ticket) && threadIdx.x < 4) {
        const unsigned long long v = __ldcg(amax_bits + threadIdx.x);
        host_out[threadIdx.x] =
            threadIdx.x < 3 ? __longlong_as_double((long long)v) : (double)v / sum_scale;
    }
}

struct CellGrid {
    Frame fr;        // origin, axes, lo[] (cell-grid origin in frame coords)
    double cell[3];  // cell size per axis
    long long n[3];  // cells per axis
    double quantum, inv_quantum;  // chunk centres are multiples of quantum (a power of two)
};

__device__ __forceinline__ void cell_of(const CellGrid& g, double x, double y, double z,
                                        long long ic[3]) {
    double c[3];
    to_frame(g.fr, x, y, z, c);
    for (int a = 0; a < 3; ++a) {
        double q = g.cell[a] > 0.0 ? floor((c[a] - g.fr.lo[a]) / g.cell[a]) : 0.0;
        long long v = (long long)q;
        v = v < 0 ? 0 : (v >= g.n[a] ? g.n[a] - 1 : v);
        ic[a] = v;
    }
}

__global__ void ray_keys_kernel(RaysDev r, int n, CellGrid g, uint64_t* __restrict__ keys,
                                int* __restrict__ idx) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    long long ic[3];
    cell_of(g, r.x[i], r.y[i], r.z[i], ic);
    keys[i] = (uint64_t)((ic[2] * g.n[1] + ic[1]) * g.n[0] + ic[0]);
    idx[i] = i;
}

__global__ void head_flags_kernel(const uint64_t* __restrict__ keys, int n, int* __restrict__ flags) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    flags[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1 : 0;
}

__global__ void chunk_table_kernel(const uint64_t* __restrict__ keys, const int* __restrict__ flags,
                                   const int* __restrict__ run_id, int n, CellGrid g,
                                   int* __restrict__ chunk_begin, double* __restrict__ chunk_center,
                                   int* __restrict__ n_chunks, int* __restrict__ host_chunks) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (flags[i]) {
        int c = run_id[i] - 1;
        chunk_begin[c] = i;
        uint64_t k = keys[i];
        long long ix = (long long)(k % (uint64_t)g.n[0]);
        long long iy = (long long)((k / (uint64_t)g.n[0]) % (uint64_t)g.n[1]);
        long long iz = (long long)(k / ((uint64_t)g.n[0] * (uint64_t)g.n[1]));
        double f0 = g.fr.lo[0] + (ix + 0.5) * g.cell[0];
        double f1 = g.fr.lo[1] + (iy + 0.5) * g.cell[1];
        double f2 = g.fr.lo[2] + (iz + 0.5) * g.cell[2];
        const Frame& fr = g.fr;
        // Snapped to multiples of g.quantum (a power of two no smaller than the
        // ulp of any coordinate in play), so that q = p - R0 is exact: at
        // |p| ~ 2e4 mm one rounding of q is 1.8e-12 mm, 2.8e-4 rad at 30 keV.
        const double cx = fr.ox + f0 * fr.e1[0] + f1 * fr.e2[0] + f2 * fr.u0[0];
        const double cy = fr.oy + f0 * fr.e1[1] + f1 * fr.e2[1] + f2 * fr.u0[1];
        const double cz = fr.oz + f0 * fr.e1[2] + f1 * fr.e2[2] + f2 * fr.u0[2];
        chunk_center[3 * c + 0] = rint(cx * g.inv_quantum) * g.quantum;
        chunk_center[3 * c + 1] = rint(cy * g.inv_quantum) * g.quantum;
        chunk_center[3 * c + 2] = rint(cz * g.inv_quantum) * g.quantum;
    }
    if (i == n - 1) {
        int nc = run_id[i];
        *n_chunks = nc;
        *host_chunks = nc;
        chunk_begin[nc] = n;
    }
}

__global__ void records_kernel(RaysDev r, int n, const int* __restrict__ sorted_idx,
                               const int* __restrict__ run_id, const double* __restrict__ chunk_center,
                               PrRawRay* __restrict__ recs) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int c = run_id[i] - 1;
    int o = sorted_idx[i];
    PrRawRay rec;
    rec.rx = r.x[o] - chunk_center[3 * c + 0];
    rec.ry = r.y[o] - chunk_center[3 * c + 1];
    rec.rz = r.z[o] - chunk_center[3 * c + 2];
    rec.es_re = (float)r.es_re[o];
    rec.es_im = (float)r.es_im[o];
    rec.ep_re = (float)r.ep_re[o];
    rec.ep_im = (float)r.ep_im[o];
    rec.nx = (float)r.nx[o];
    rec.ny = (float)r.ny[o];
    rec.nz = (float)r.nz[o];
    rec.nl = (float)r.nl[o];
    rec.pad0 = rec.pad1 = 0.f;
    recs[i] = rec;
}

// Orders the ray groups of a solve by decreasing estimated cost, so that the
// persistent kernel hands out the most expensive (tile, group) items first and
// the launch does not end on a few long ones. A group's cost is its ray count
// plus kGroupChunkCost rays for every chunk it spans (each chunk boundary
// costs a per-point set-up and flush, about the sweep of that many rays).
// One block, bitonic sort of (cost, group) keys in shared memory; ties keep
// group order, so the schedule is deterministic. groups <= kMaxGroups.
constexpr int kMaxGroups = 4096;
constexpr int kGroupChunkCost = 24;

__global__ void __launch_bounds__(1024) group_order_kernel(const int* __restrict__ chunk_begin,
                                                           const int* __restrict__ n_chunks_dev,
                                                           int n, int groups,
                                                           int* __restrict__ order) {
    __shared__ unsigned long long key[kMaxGroups];
    const int n_chunks = *n_chunks_dev;
    int len = 1;
    while (len < groups) len <<= 1;
    auto chunk_at = [&](int pos) {
        int lo = 0, hi = n_chunks - 1;
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (chunk_begin[mid] <= pos) lo = mid;
            else hi = mid - 1;
        }
        return lo;
    };
    for (int g = threadIdx.x; g < len; g += blockDim.x) {
        unsigned long long k = ~0ull;
        if (g < groups) {
            const long long r0 = (long long)g * n / groups, r1 = (long long)(g + 1) * n / groups;
            unsigned int cost = 0;
            if (r1 > r0) {
                const int c = chunk_at((int)(r1 - 1)) - chunk_at((int)r0) + 1;
                const long long w = (r1 - r0) + (long long)kGroupChunkCost * c;
                cost = (unsigned int)(w < 0x7fffffffLL ? w : 0x7fffffffLL);
            }
            // Ascending keys = descending cost, then ascending group.
            k = ((unsigned long long)(0xffffffffu - cost) << 32) | (unsigned int)g;
        }
        key[g] = k;
    }
    __syncthreads();
    for (int size = 2; size <= len; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = threadIdx.x; i < len; i += blockDim.x) {
                const int j = i ^ stride;
                if (j > i) {
                    const bool up = (i & size) == 0;
                    const unsigned long long a = key[i], b = key[j];
                    if ((a > b) == up) {
                        key[i] = b;
                        key[j] = a;
                    }
                }
            }
            __syncthreads();
        }
    for (int i = threadIdx.x; i < groups; i += blockDim.x) order[i] = (int)(key[i] & 0xffffffffu);
}

// Adds the groups' slots of every tile slot and scatters the sum to the screen
// point's original index: a block takes kFinSlots slots, its kFinLanes rows of
// threads every kFinLanes-th group each (with one row a line of 256 points and
// 44 groups took 31 us, one dependent load after the other), and row 0 adds the
// rows in order. One-polarization solves hold A in components 0 and 1; the
// field is (pes * A, pep * A).
constexpr int kFinSlots = 32, kFinLanes = 16;

__global__ void __launch_bounds__(kFinSlots * kFinLanes)
finalize_kernel(const double* __restrict__ partial, const int* __restrict__ tile_perm, int groups,
                int slots, FieldDev out, int one_pol, double2 pes, double2 pep) {
    __shared__ double sm[kFinLanes][4][kFinSlots];
    const int x = threadIdx.x % kFinSlots, y = threadIdx.x / kFinSlots;
    const int s = blockIdx.x * kFinSlots + x;  // slots is a multiple of 256
    const int nc = one_pol ? 2 : 4;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
    for (int g = y; g < groups; g += kFinLanes) {
        const double* b = partial + (size_t)g * 4 * slots;
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (c < nc) acc[c] += b[(size_t)c * slots + s];
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) sm[y][c][x] = acc[c];
    __syncthreads();
    if (y != 0) return;
    const int id = tile_perm[s];
    if (id < 0) return;
#pragma unroll
    for (int c = 0; c < 4; ++c)
        for (int w = 1; w < kFinLanes; ++w) acc[c] += sm[w][c][x];
    if (one_pol) {
        out.es_re[id] = pes.x * acc[0] - pes.y * acc[1];
        out.es_im[id] = pes.x * acc[1] + pes.y * acc[0];
        out.ep_re[id] = pep.x * acc[0] - pep.y * acc[1];
        out.ep_im[id] = pep.x * acc[1] + pep.y * acc[0];
        return;
    }
    out.es_re[id] = acc[0];
    out.es_im[id] = acc[1];
    out.ep_re[id] = acc[2];
    out.ep_im[id] = acc[3];
}

// ---------------------------------------------------------------------------
// Persistent kernel
// ---------------------------------------------------------------------------

using namespace sm100;  // mbarriers with bounded waits, bulk copies (xk_sm100.cuh)

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Error-free sum of hi and x into (hi, lo) (Knuth's TwoSum).
__device__ __forceinline__ void two_sum_acc(float& hi, float& lo, float x) {
    float s = hi + x;
    float bb = s - hi;
    float err = (hi - (s - bb)) + (x - bb);
    hi = s;
    lo += err;
}

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }

// Prepared record in shared memory (in place of the 64-byte raw record):
//   a = {rho_x, rho_y, rho_z, R = k |rho_perp|^2}
//   b = {W = -2 u.rho, G = -2 n.rho, nl, -W}
//   e = {es', ep'} with the per-ray phasor exp(-i k u.rho) applied
//   n = {2 nx, 2 ny, 2 nz, 0}
//
// Per-warp shared state besides the two ray buffers. NC components per point:
// 4 (Es, Ep) or 2 (the one-polarization kernels' single column), which is
// what lets those kernels fit four CTAs per SM.
template <bool FOLD>
struct ChunkGeometry {        // unfolded: of the current chunk
    float2 ph[kPrPpl][32];    // (k/2pi) i exp(i k |q|)
    double ux, uy, uz;        // item direction
    double r0x, r0y, r0z;     // chunk centre
};
// Folded kernels switch chunks every few dozen rays: lane l prepares chunk
// first + l of the next 32 at once. Q = tile centre - chunk centre, D = |Q|.
//   dir   u = Q / D
//   geo   flat tiles: 1 / (2 D), 2 / D, frac(k D / 2 pi); others: chunk centre
//   geof  flat tiles: 1 / D, 1 / (2 D) or 2 D (SFU sweep) as hi + lo, 2 n.Q, Q
template <>
struct ChunkGeometry<true> {
    double dir[3][32], geo[3][32];
    float geof[7][32];
};
template <int NC, bool FOLD>
struct WarpSharedT : ChunkGeometry<FOLD> {
    static constexpr int kNC = NC;
    float hi[kPrPpl * NC][32];  // two-float accumulators, [point*NC + component][lane]
    float lo[kPrPpl * NC][32];
    uint64_t bar[2];            // mbarriers of the two ray buffers
};

// Per-lane state of the SFU sweep.
template <bool UNIFORM>
struct ScalarState {
    float vx[kPrPpl], vy[kPrPpl], vz[kPrPpl], q2[kPrPpl];  // q2 = 2|q|
    float nq[kPrPpl];                                        // 2 n.q (UNIFORM)
    float qx[kPrPpl], qy[kPrPpl], qz[kPrPpl];                // q (general normals)
    float phi[kPrPpl];                                       // base phase k|q| mod 2 pi
    float acc[kPrPpl][4];
};

// Per-lane state of the packed sweep: point pairs (2i, 2i+1).
template <bool UNIFORM>
struct PackedState {
    float2 vx[kPrPpl / 2], vy[kPrPpl / 2], vz[kPrPpl / 2], q2[kPrPpl / 2];  // q2 = 1/(2|q|)
    float2 nq[kPrPpl / 2];
    float2 qx[kPrPpl / 2], qy[kPrPpl / 2], qz[kPrPpl / 2];
    float2 phi[kPrPpl / 2];  // base phase k|q| mod 2 pi
    float2 acc[kPrPpl / 2][4];
};

// Per chunk: FP64 geometry of the lane's points, written into the sweep
// state, and the per-point base phase k|q|: folded into the sweep state
// (FOLD) or as the chunk phasor (k/2pi) i exp(i k|q|) into shared memory.
template <bool UNIFORM, bool FAST, bool FOLD, class State, class WS>
__device__ __forceinline__ void setup_points(const PrSolve& sv, int t, int lane, WS& ws,
                                             State& st, double ux, double uy, double uz,
                                             double r0x, double r0y, double r0z) {
    const double k = sv.k;
    float* vxp = reinterpret_cast<float*>(st.vx);
    float* vyp = reinterpret_cast<float*>(st.vy);
    float* vzp = reinterpret_cast<float*>(st.vz);
    float* q2p = reinterpret_cast<float*>(st.q2);
    float* nqp = reinterpret_cast<float*>(st.nq);
    float* qxp = reinterpret_cast<float*>(st.qx);
    float* qyp = reinterpret_cast<float*>(st.qy);
    float* qzp = reinterpret_cast<float*>(st.qz);
#pragma unroll
    for (int i = 0; i < kPrPpl; ++i) {
        const long long s = (long long)t * kPrTile + lane + 32 * i;
        double qx = sv.tpx[s] - r0x, qy = sv.tpy[s] - r0y, qz = sv.tpz[s] - r0z;
        // Base phase k|q| in turns, carried in double-double (k|q| reaches
        // 1e12 rad at 30 keV and 20 m, where one FP64 rounding is 1e-4 rad);
        // the same square root gives |q|.
        double qn, inv2q;
        const float fr = (float)dd_turns(sv.kt, sv.kt_lo, qx, qy, qz, &qn, &inv2q);
        double vx = qx - qn * ux, vy = qy - qn * uy, vz = qz - qn * uz;
        vxp[i] = (float)(-2.0 * k * vx);
        vyp[i] = (float)(-2.0 * k * vy);
        vzp[i] = (float)(-2.0 * k * vz);
        q2p[i] = FAST ? (float)inv2q : (float)(2.0 * qn);
        if (UNIFORM) {
            nqp[i] = (float)(2.0 * ((double)sv.unx * qx + (double)sv.uny * qy + (double)sv.unz * qz));
        } else {
            qxp[i] = (float)qx;
            qyp[i] = (float)qy;
            qzp[i] = (float)qz;
        }
        if (FOLD) {
            // The base phase enters the FP32 residual phase of every pair of
            // the chunk (|fr| <= 1/2 turn), so the chunk sums need no phasor.
            reinterpret_cast<float*>(st.phi)[i] = 6.28318530717958647692f * fr;
        } else {
            // |fr| <= 1/2 turn: the SFU sin/cos is accurate to ~5e-7 on [-pi, pi].
            const float kt = (float)sv.kt;
            float sp, cp;
            __sincosf(6.28318530717958647692f * fr, &sp, &cp);
            if constexpr (!FOLD) ws.ph[i][lane] = make_float2(-kt * sp, kt * cp);
        }
    }
}

// Folded kernels: geometry of chunks first .. first + 31 (clamped to the last).
template <bool UNIFORM, bool FAST, class WS>
__device__ __forceinline__ void chunk_geometry(const PrSolve& sv, int t, int first, int n_chunks,
                                               int lane, WS& ws) {
    const int c = min(first + lane, n_chunks - 1);
    const double rx = sv.chunk_center[3 * c], ry = sv.chunk_center[3 * c + 1],
                 rz = sv.chunk_center[3 * c + 2];
    const double qx = sv.tile_center[3 * t] - rx, qy = sv.tile_center[3 * t + 1] - ry,
                 qz = sv.tile_center[3 * t + 2] - rz;
    if (!sv.flat) {
        const double inv = 1.0 / sqrt(qx * qx + qy * qy + qz * qz);
        ws.dir[0][lane] = qx * inv;
        ws.dir[1][lane] = qy * inv;
        ws.dir[2][lane] = qz * inv;
        ws.geo[0][lane] = rx;
        ws.geo[1][lane] = ry;
        ws.geo[2][lane] = rz;
        return;
    }
    double d, unused;
    const double turns = dd_turns(sv.kt, sv.kt_lo, qx, qy, qz, &d, &unused);
    const double inv = 1.0 / d, ux = qx * inv, uy = qy * inv, uz = qz * inv;
    ws.dir[0][lane] = ux;
    ws.dir[1][lane] = uy;
    ws.dir[2][lane] = uz;
    ws.geo[0][lane] = 0.5 * inv;
    ws.geo[1][lane] = 2.0 * inv;
    ws.geo[2][lane] = turns - rint(turns);
    ws.geof[0][lane] = (float)inv;
    const double base = FAST ? 0.5 * inv : 2.0 * d;
    ws.geof[1][lane] = (float)base;
    ws.geof[2][lane] = (float)(base - (double)(float)base);
    if (UNIFORM)
        ws.geof[3][lane] =
            (float)(2.0 * ((double)sv.unx * qx + (double)sv.uny * qy + (double)sv.unz * qz));
    ws.geof[4][lane] = (float)qx;
    ws.geof[5][lane] = (float)qy;
    ws.geof[6][lane] = (float)qz;
}

// The set-up of a flat tile's points: |q| expanded about the tile centre.
// With s = p - tile centre, h = u.s + s^2 / (2D) and e = 2 h / D,
//     |q| - D = h (1 - e/4 + e^2/8 - 5 e^3/64 + 7 e^4/128 - ...),
// whose product with k / 2 pi (1e4 turns) needs FP64 but no double-double, and
// v = s - (|q| - D) u. 14 FP64 operations per point instead of 55.
template <bool UNIFORM, bool FAST, class State, class WS>
__device__ __forceinline__ void setup_points_flat(const PrSolve& sv, int t, int lane, const WS& ws,
                                                  int g, State& st) {
    float* vxp = reinterpret_cast<float*>(st.vx);
    float* vyp = reinterpret_cast<float*>(st.vy);
    float* vzp = reinterpret_cast<float*>(st.vz);
    float* q2p = reinterpret_cast<float*>(st.q2);
    float* nqp = reinterpret_cast<float*>(st.nq);
    float* qxp = reinterpret_cast<float*>(st.qx);
    float* qyp = reinterpret_cast<float*>(st.qy);
    float* qzp = reinterpret_cast<float*>(st.qz);
    float* php = reinterpret_cast<float*>(st.phi);
    const double ux = ws.dir[0][g], uy = ws.dir[1][g], uz = ws.dir[2][g];
    const double half_inv = ws.geo[0][g], two_inv = ws.geo[1][g], turn0 = ws.geo[2][g];
    const float inv = ws.geof[0][g], base = ws.geof[1][g], base_lo = ws.geof[2][g];
    const double kt = sv.kt, m2k = -2.0 * sv.k;
    constexpr double kRound = 6755399441055744.0;  // 1.5 * 2^52
#pragma unroll
    for (int i = 0; i < kPrPpl; ++i) {
        const size_t s = (size_t)t * kPrTile + lane + 32 * i;
        const double4 r = sv.tile_rel[s];
        const double h = fma(r.w, half_inv, fma(uz, r.z, fma(uy, r.y, ux * r.x)));
        const double e = h * two_inv;
        double p = fma(e, 7.0 / 128.0, -5.0 / 64.0);
        p = fma(e, p, 0.125);
        p = fma(e, p, -0.25);
        const double d = fma(h * e, p, h);
        const double w = fma(kt, d, turn0);
        php[i] = 6.28318530717958647692f * (float)(w - ((w + kRound) - kRound));
        const float df = (float)d;
        // In FP64: with FP32 offsets the error of the near-field screen rose from
        // 7.6e-6 to 8.1e-6, and tenfold on tiles that reach along u.
        vxp[i] = (float)(m2k * fma(-d, ux, r.x));
        vyp[i] = (float)(m2k * fma(-d, uy, r.y));
        vzp[i] = (float)(m2k * fma(-d, uz, r.z));
        const float x = df * inv;
        // One rounding, as (float)(1 / (2 |q|)) has: an error here is shared by
        // every pair of the point and the chunk.
        q2p[i] = base + (FAST ? fmaf(base, x * (x - 1.f), base_lo) : fmaf(2.f, df, base_lo));
        if (UNIFORM) {
            nqp[i] = ws.geof[3][g] + sv.tile_ns[s];
        } else {
            qxp[i] = ws.geof[4][g] + (float)r.x;
            qyp[i] = ws.geof[5][g] + (float)r.y;
            qzp[i] = ws.geof[6][g] + (float)r.z;
        }
    }
}

// Unfolded variants, at every chunk boundary and at the item end: multiplies
// the lane's two-float chunk sums by the chunk phasor in FP64, adds them to
// the item's slots (tile-slot order) and clears the sums.
template <bool POL, class WS>
__device__ __forceinline__ void flush_chunk(const PrSolve& sv, int t, int g, int lane, WS& ws) {
    constexpr int NC = WS::kNC;
    const size_t slots = (size_t)sv.n_tiles * kPrTile;
    double* base = sv.partial + (size_t)g * 4 * slots;
#pragma unroll 2
    for (int i = 0; i < kPrPpl; ++i) {
        const size_t s = (size_t)t * kPrTile + lane + 32 * i;
        const float2 ph = ws.ph[i][lane];
        const double phr = ph.x, phi = ph.y;
        double v[4];
#pragma unroll
        for (int c = 0; c < (POL ? 2 : 4); ++c) {
            v[c] = (double)ws.hi[i * NC + c][lane] + (double)ws.lo[i * NC + c][lane];
            ws.hi[i * NC + c][lane] = 0.f;
            ws.lo[i * NC + c][lane] = 0.f;
        }
        // Each slot is updated by this one thread, in chunk order; the atomic
        // form only lets the warp go on without waiting for the loads.
        atomicAdd(base + 0 * slots + s, v[0] * phr - v[1] * phi);
        atomicAdd(base + 1 * slots + s, v[0] * phi + v[1] * phr);
        if (!POL) {
            atomicAdd(base + 2 * slots + s, v[2] * phr - v[3] * phi);
            atomicAdd(base + 3 * slots + s, v[2] * phi + v[3] * phr);
        }
    }
}

// Folded variants, once at the item end: multiplies the lane's two-float
// sums of the item by i k / (2 pi) in FP64 and adds them to the item's slots.
template <bool POL, class WS>
__device__ __forceinline__ void flush_item(const PrSolve& sv, int t, int g, int lane, WS& ws) {
    constexpr int NC = WS::kNC;
    const size_t slots = (size_t)sv.n_tiles * kPrTile;
    double* base = sv.partial + (size_t)g * 4 * slots;
    const double kt = sv.kt;
#pragma unroll 2
    for (int i = 0; i < kPrPpl; ++i) {
        const size_t s = (size_t)t * kPrTile + lane + 32 * i;
        double v[4];
#pragma unroll
        for (int c = 0; c < (POL ? 2 : 4); ++c)
            v[c] = (double)ws.hi[i * NC + c][lane] + (double)ws.lo[i * NC + c][lane];
        // Sub-items of one (group, tile) add into the same slots in sub
        // order (never two in one launch); the atomic form only lets the warp
        // go on without waiting for the loads.
        atomicAdd(base + 0 * slots + s, -kt * v[1]);
        atomicAdd(base + 1 * slots + s, kt * v[0]);
        if (!POL) {
            atomicAdd(base + 2 * slots + s, -kt * v[3]);
            atomicAdd(base + 3 * slots + s, kt * v[2]);
        }
    }
}

// Prepares the stage's rays for the item direction (lane j handles rays
// j, j+32).
// One-polarization kernels (POL) prepare the one amplitude column they sum;
// the unfolded ones (POLAR) keep it in polar form, e = {|a|, psi}, psi the
// amplitude's phase plus the ray phase -k u.rho, which the sweep adds to the
// pair's residual phase inside the FMA that forms it, so that a pair costs
// one multiply and two FMAs on the sums instead of a complex multiply-add.
// (In the folded kernels the same form measured 3x the field error and no
// faster; they keep the Cartesian amplitude.)
template <bool POL, bool POLAR>
__device__ __forceinline__ void prep_stage(PrRawRay* buf, int len, int lane, const PrSolve& sv,
                                           double ux, double uy, double uz) {
    for (int j = lane; j < len; j += 32) {
        const PrRawRay r = buf[j];
        double ur = ux * r.rx + uy * r.ry + uz * r.rz;
        double tx = r.rx - ur * ux, ty = r.ry - ur * uy, tz = r.rz - ur * uz;
        double perp2 = tx * tx + ty * ty + tz * tz;
        double turns = -sv.kt * ur;
        float f = (float)(turns - rint(turns));
        float sn = 0.f, cs = 1.f;
        if (!POLAR) __sincosf(6.28318530717958647692f * f, &sn, &cs);
        float rxf = (float)r.rx, ryf = (float)r.ry, rzf = (float)r.rz;
        float w = (float)(-2.0 * ur);
        float4 a = make_float4(rxf, ryf, rzf, (float)(sv.k * perp2));
        float4 b = make_float4(w, -2.f * (r.nx * rxf + r.ny * ryf + r.nz * rzf), r.nl, -w);
        float4 e;
        if (POLAR) {
            const float pr = sv.amp_src ? r.ep_re : r.es_re, pi = sv.amp_src ? r.ep_im : r.es_im;
            // |psi| <= 2 pi: f in [-1/2, 1/2] turns, atan2 in [-pi, pi].
            e = make_float4(hypotf(pr, pi), fmaf(6.28318530717958647692f, f, atan2f(pi, pr)),
                            0.f, 0.f);
        } else if (POL) {
            const float pr = sv.amp_src ? r.ep_re : r.es_re, pi = sv.amp_src ? r.ep_im : r.es_im;
            e = make_float4(pr * cs - pi * sn, pr * sn + pi * cs, 0.f, 0.f);
        } else {
            e = make_float4(r.es_re * cs - r.es_im * sn, r.es_re * sn + r.es_im * cs,
                            r.ep_re * cs - r.ep_im * sn, r.ep_re * sn + r.ep_im * cs);
        }
        float4 nn = make_float4(2.f * r.nx, 2.f * r.ny, 2.f * r.nz, 0.f);
        float4* o = reinterpret_cast<float4*>(buf + j);
        o[0] = a;
        o[1] = b;
        o[2] = e;
        o[3] = nn;
    }
}

// Adds the lane's FP32 partials into its two-float accumulators and clears
// them (after every stage, that is at most kPrStage rays of one chunk).
// One-polarization kernels (POL) carry components 0 and 1 only.
template <bool POL, bool UNIFORM, class WS>
__device__ __forceinline__ void fold_acc(ScalarState<UNIFORM>& ls, WS& ws, int lane) {
    constexpr int NC = WS::kNC;
#pragma unroll
    for (int i = 0; i < kPrPpl; ++i)
#pragma unroll
        for (int c = 0; c < (POL ? 2 : 4); ++c) {
            float hi = ws.hi[i * NC + c][lane], lo = ws.lo[i * NC + c][lane];
            two_sum_acc(hi, lo, ls.acc[i][c]);
            ws.hi[i * NC + c][lane] = hi;
            ws.lo[i * NC + c][lane] = lo;
            ls.acc[i][c] = 0.f;
        }
}

template <bool POL, bool UNIFORM, class WS>
__device__ __forceinline__ void fold_acc(PackedState<UNIFORM>& ls, WS& ws, int lane) {
    constexpr int NC = WS::kNC;
#pragma unroll
    for (int i = 0; i < kPrPpl / 2; ++i)
#pragma unroll
        for (int c = 0; c < (POL ? 2 : 4); ++c) {
            const float2 v = ls.acc[i][c];
            float hi0 = ws.hi[(2 * i) * NC + c][lane], lo0 = ws.lo[(2 * i) * NC + c][lane];
            float hi1 = ws.hi[(2 * i + 1) * NC + c][lane], lo1 = ws.lo[(2 * i + 1) * NC + c][lane];
            two_sum_acc(hi0, lo0, v.x);
            two_sum_acc(hi1, lo1, v.y);
            ws.hi[(2 * i) * NC + c][lane] = hi0;
            ws.lo[(2 * i) * NC + c][lane] = lo0;
            ws.hi[(2 * i + 1) * NC + c][lane] = hi1;
            ws.lo[(2 * i + 1) * NC + c][lane] = lo1;
            ls.acc[i][c] = f2(0.f);
        }
}

template <bool UNIFORM>
__device__ __forceinline__ void clear_acc(ScalarState<UNIFORM>& ls) {
#pragma unroll
    for (int i = 0; i < kPrPpl; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) ls.acc[i][c] = 0.f;
}

template <bool UNIFORM>
__device__ __forceinline__ void clear_acc(PackedState<UNIFORM>& ls) {
#pragma unroll
    for (int i = 0; i < kPrPpl / 2; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) ls.acc[i][c] = f2(0.f);
}

// SFU sweep: one point per FP32 instruction, rcp.approx for the reciprocal
// (LIN does not apply).
template <bool UNIFORM, bool FOLD, bool POL, bool LIN, class WS>
__device__ __forceinline__ void sweep_stage(const PrRawRay* buf, int len, int lane,
                                            ScalarState<UNIFORM>& ls, WS& ws) {
    const float4* rec = reinterpret_cast<const float4*>(buf);
#pragma unroll 1
    for (int j = 0; j < len; ++j) {
        const float4 a = rec[4 * j + 0];
        const float4 b = rec[4 * j + 1];
        const float4 e = rec[4 * j + 2];
        float4 nn = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!UNIFORM) nn = rec[4 * j + 3];
#pragma unroll
        for (int i = 0; i < kPrPpl; ++i) {
            float num = fmaf(ls.vx[i], a.x, a.w);
            num = fmaf(ls.vy[i], a.y, num);
            num = fmaf(ls.vz[i], a.z, num);
            const float rd = rcp_approx(ls.q2[i] + b.x);
            // One column, unfolded: the amplitude's phase e.y joins the
            // residual phase inside the FMA that forms it.
            constexpr bool POLAR = POL && !FOLD;
            const float th = FOLD ? fmaf(num, rd, ls.phi[i]) : (POLAR ? fmaf(num, rd, e.y) : num * rd);
            float sn, cs;
            __sincosf(th, &sn, &cs);
            float gq;
            if (UNIFORM) {
                gq = ls.nq[i] + b.y;
            } else {
                gq = fmaf(nn.x, ls.qx[i], fmaf(nn.y, ls.qy[i], fmaf(nn.z, ls.qz[i], b.y)));
            }
            const float obl = fmaf(gq, rd, b.z);
            const float amp = obl * rd;
            if (POLAR) {
                const float m = amp * e.x;
                ls.acc[i][0] = fmaf(m, cs, ls.acc[i][0]);
                ls.acc[i][1] = fmaf(m, sn, ls.acc[i][1]);
                continue;
            }
            const float ac = amp * cs, as = amp * sn;
            ls.acc[i][0] = fmaf(e.x, ac, fmaf(-e.y, as, ls.acc[i][0]));
            ls.acc[i][1] = fmaf(e.x, as, fmaf(e.y, ac, ls.acc[i][1]));
            if (!POL) {
                ls.acc[i][2] = fmaf(e.z, ac, fmaf(-e.w, as, ls.acc[i][2]));
                ls.acc[i][3] = fmaf(e.z, as, fmaf(e.w, ac, ls.acc[i][3]));
            }
        }
    }
}

// Packed sweep: two points per f32x2 instruction, series reciprocal
// r0 (1 + e + e^2), or r0 (1 + e) when the planner bounds |e|^2 times the
// phase budget far below the tolerance (LIN: one f32x2 FMA fewer per pair of
// points).
template <bool UNIFORM, bool FOLD, bool POL, bool LIN, class WS>
__device__ __forceinline__ void sweep_stage(const PrRawRay* buf, int len, int lane,
                                            PackedState<UNIFORM>& ls, WS& ws) {
    constexpr int H = kPrPpl / 2;
    const float4* rec = reinterpret_cast<const float4*>(buf);
    // Two rays per iteration give the scheduler two independent sets of
    // chains (+3 % one-column, +1 % two-column on the far-field workload).
    // The folded (near-field) kernels switch chunks every few stages and ran
    // ~5 % slower unrolled; they and the general-normal two-column kernels,
    // which are at the register limit of three CTAs per SM, keep one.
#pragma unroll (((UNIFORM || POL) && !FOLD) ? 2 : 1)
    for (int j = 0; j < len; ++j) {
        const float4 a = rec[4 * j + 0];
        const float4 b = rec[4 * j + 1];
        const float4 e = rec[4 * j + 2];
        float4 nn = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!UNIFORM) nn = rec[4 * j + 3];
        const float2 ax = f2(a.x), ay = f2(a.y), az = f2(a.z), aw = f2(a.w);
        const float2 wn = f2(b.w), gg = f2(b.y), nl = f2(b.z);
        const float2 ex = f2(e.x), ey = f2(e.y), ez = f2(e.z), ew = f2(e.w);
        const float2 ney = f2(-e.y), new_ = f2(-e.w);
#pragma unroll
        for (int i = 0; i < H; ++i) {
            float2 num = __ffma2_rn(ls.vx[i], ax, aw);
            num = __ffma2_rn(ls.vy[i], ay, num);
            num = __ffma2_rn(ls.vz[i], az, num);
            // 1/(2|q| - 2u.rho) = r0 / (1 - e), e = 2u.rho r0 ~ r0 (1 + e + e^2)
            const float2 ep = __fmul2_rn(wn, ls.q2[i]);
            const float2 rd = LIN ? __ffma2_rn(ls.q2[i], ep, ls.q2[i])
                                  : __ffma2_rn(ls.q2[i], __ffma2_rn(ep, ep, ep), ls.q2[i]);
            constexpr bool POLAR = POL && !FOLD;
            const float2 th = FOLD ? __ffma2_rn(num, rd, ls.phi[i])
                                   : (POLAR ? __ffma2_rn(num, rd, ey) : __fmul2_rn(num, rd));
            float s0, c0, s1, c1;
            __sincosf(th.x, &s0, &c0);
            __sincosf(th.y, &s1, &c1);
            float2 gq;
            if (UNIFORM) {
                gq = __fadd2_rn(ls.nq[i], gg);
            } else {
                gq = __ffma2_rn(f2(nn.x), ls.qx[i],
                                __ffma2_rn(f2(nn.y), ls.qy[i], __ffma2_rn(f2(nn.z), ls.qz[i], gg)));
            }
            const float2 obl = __ffma2_rn(gq, rd, nl);
            const float2 amp = __fmul2_rn(obl, rd);
            if (POLAR) {
                const float2 m = __fmul2_rn(amp, ex);
                ls.acc[i][0] = __ffma2_rn(m, f2(c0, c1), ls.acc[i][0]);
                ls.acc[i][1] = __ffma2_rn(m, f2(s0, s1), ls.acc[i][1]);
                continue;
            }
            const float2 ac = __fmul2_rn(amp, f2(c0, c1));
            const float2 as = __fmul2_rn(amp, f2(s0, s1));
            ls.acc[i][0] = __ffma2_rn(ex, ac, __ffma2_rn(ney, as, ls.acc[i][0]));
            ls.acc[i][1] = __ffma2_rn(ex, as, __ffma2_rn(ey, ac, ls.acc[i][1]));
            if (!POL) {
                ls.acc[i][2] = __ffma2_rn(ez, ac, __ffma2_rn(new_, as, ls.acc[i][2]));
                ls.acc[i][3] = __ffma2_rn(ez, as, __ffma2_rn(ew, ac, ls.acc[i][3]));
            }
        }
    }
}

struct WarpPipe {
    PrRawRay* buf[2];
    uint64_t* bar[2];
    uint32_t phase;  // bit b: parity of the next completion of buffer b
};

// `extra` bytes beyond the copy are expected only by the stall test hook
// (PrCtl::stall_bytes); 0 otherwise.
__device__ __forceinline__ void issue_stage(WarpPipe& wp, int b, const PrRawRay* src, int len,
                                            int lane, uint32_t extra = 0) {
    if (lane == 0) {
        uint32_t bytes = (uint32_t)len * (uint32_t)sizeof(PrRawRay);
        mbar_arrive_expect_tx(wp.bar[b], bytes + extra);
        bulk_g2s(wp.buf[b], src, bytes, wp.bar[b]);
    }
}

__device__ __forceinline__ int chunk_of(const int* __restrict__ begin, int n_chunks, int pos) {
    int lo = 0, hi = n_chunks - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (begin[mid] <= pos) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Processes one (tile, ray-range) item; false if a bounded wait ran out.
template <bool UNIFORM, bool FAST, bool FOLD, bool POL, bool LIN>
__device__ bool process_item(const PrSolve& sv, long long local, WarpPipe& wp,
                             WarpSharedT<POL ? 2 : 4, FOLD>& ws,
                             int lane, uint32_t wait_limit, uint32_t stall_bytes) {
    // local = (sub * groups + g) * n_tiles + t: sub-range `sub` of ray group g
    // against tile t. Sub-items of one (g, t) add into the same slots, so a
    // launch must never hold two of them (launches cover at most
    // groups * n_tiles consecutive items of a solve).
    const int t = (int)(local % sv.n_tiles);
    const long long rest = local / sv.n_tiles;
    const int rank = (int)(rest % sv.groups);
    const int g = sv.group_order ? sv.group_order[rank] : rank;
    const int sub = (int)(rest / sv.groups);
    const long long n = sv.n_rays;
    const long long g0 = (long long)g * n / sv.groups;
    const long long g1 = (long long)(g + 1) * n / sv.groups;
    const int r0 = (int)(g0 + (g1 - g0) * sub / sv.subs);
    const int r1 = (int)(g0 + (g1 - g0) * (sub + 1) / sv.subs);
    if (r0 >= r1) return true;
    const int n_chunks = *sv.n_chunks_dev;
    const int* __restrict__ cb = sv.chunk_begin;

#pragma unroll
    for (int i = 0; i < kPrPpl * (POL ? 2 : 4); ++i) ws.hi[i][lane] = ws.lo[i][lane] = 0.f;

    using State = typename std::conditional<FAST, PackedState<UNIFORM>, ScalarState<UNIFORM>>::type;
    State st;
    clear_acc(st);
    int cur_chunk = -1;
    int geo_first = -64;  // FOLD: first of the 32 chunks whose geometry is in `ws`
    int pos = r0;
    int c = chunk_of(cb, n_chunks, pos);
    int len = min(kPrStage, min(cb[c + 1], r1) - pos);
    int b = 0;
    issue_stage(wp, b, sv.recs + pos, len, lane, stall_bytes);
    while (true) {
        // Next stage: same chunk, or the next one at a chunk boundary.
        const int npos = pos + len;
        int nc = c;
        int nlen = 0;
        if (npos < r1) {
            if (npos >= cb[c + 1]) nc = c + 1;
            nlen = min(kPrStage, min(cb[nc + 1], r1) - npos);
            issue_stage(wp, b ^ 1, sv.recs + npos, nlen, lane);
        }
        const uint32_t par = (wp.phase >> b) & 1u;
        const bool ok = mbar_wait(wp.bar[b], par, wait_limit);
        wp.phase ^= (1u << b);
        if (!ok) {
            // Before the warp leaves, give both buffers' copies another
            // bounded wait, so that none is still writing into this warp's
            // shared memory when the block exits: this stage's (a slow copy
            // lands; a barrier that can never complete runs out again) and
            // the next stage's, already issued.
            mbar_wait(wp.bar[b], par, wait_limit);
            if (nlen > 0) {
                mbar_wait(wp.bar[b ^ 1], (wp.phase >> (b ^ 1)) & 1u, wait_limit);
                wp.phase ^= (1u << (b ^ 1));
            }
            return false;
        }
        if (c != cur_chunk) {
            if constexpr (FOLD) {
                if (c - geo_first >= 32) {
                    geo_first = c;
                    __syncwarp();
                    chunk_geometry<UNIFORM, FAST>(sv, t, c, n_chunks, lane, ws);
                    __syncwarp();
                }
                const int gi = c - geo_first;
                if (sv.flat)
                    setup_points_flat<UNIFORM, FAST>(sv, t, lane, ws, gi, st);
                else
                    setup_points<UNIFORM, FAST, FOLD>(sv, t, lane, ws, st, ws.dir[0][gi],
                                                      ws.dir[1][gi], ws.dir[2][gi], ws.geo[0][gi],
                                                      ws.geo[1][gi], ws.geo[2][gi]);
            } else {
                if (cur_chunk >= 0) flush_chunk<POL>(sv, t, g, lane, ws);
                __syncwarp();
                if (lane == 0) {
                    const double p0x = sv.tile_center[3 * t], p0y = sv.tile_center[3 * t + 1],
                                 p0z = sv.tile_center[3 * t + 2];
                    const double r0x = sv.chunk_center[3 * c], r0y = sv.chunk_center[3 * c + 1],
                                 r0z = sv.chunk_center[3 * c + 2];
                    const double dx = p0x - r0x, dy = p0y - r0y, dz = p0z - r0z;
                    const double inv = 1.0 / sqrt(dx * dx + dy * dy + dz * dz);
                    ws.ux = dx * inv;
                    ws.uy = dy * inv;
                    ws.uz = dz * inv;
                    ws.r0x = r0x;
                    ws.r0y = r0y;
                    ws.r0z = r0z;
                }
                __syncwarp();
                setup_points<UNIFORM, FAST, FOLD>(sv, t, lane, ws, st, ws.ux, ws.uy, ws.uz, ws.r0x,
                                                  ws.r0y, ws.r0z);
            }
            cur_chunk = c;
        }
        if constexpr (FOLD) {
            const int gi = c - geo_first;
            prep_stage<POL, false>(wp.buf[b], len, lane, sv, ws.dir[0][gi], ws.dir[1][gi],
                                   ws.dir[2][gi]);
        } else {
            prep_stage<POL, POL>(wp.buf[b], len, lane, sv, ws.ux, ws.uy, ws.uz);
        }
        __syncwarp();
        sweep_stage<UNIFORM, FOLD, POL, LIN>(wp.buf[b], len, lane, st, ws);
        // FP32 partials hold one stage of one chunk. (Over several short chunks they
        // saved 8 % between mirrors, 2.6 % on the near-field screen, and cost a tenth of
        // the error between mirrors: 3.7e-7 instead of 3.3e-7.)
        fold_acc<POL>(st, ws, lane);
        // Order this stage's generic-proxy accesses before the next bulk
        // copy into the same buffer.
        fence_proxy_async();
        __syncwarp();
        if (nlen == 0) break;
        pos = npos;
        c = nc;
        len = nlen;
        b ^= 1;
    }
    if constexpr (FOLD) flush_item<POL>(sv, t, g, lane, ws);
    else flush_chunk<POL>(sv, t, g, lane, ws);
    __syncwarp();
    return true;
}

// Every solve in `solves` must match the kernel's variant (normal mode and
// sweep); solves[s].item_begin is the prefix sum of the item counts in this
// launch, and the launch covers items [item_offset, item_offset + count) of
// each solve.
template <bool UNIFORM, bool FAST, bool FOLD, bool POL, bool LIN>
__global__ void __launch_bounds__(kPrWarpsPerCta * 32, (POL && !FOLD) ? 4 : 3)
pr_persistent_kernel(const PrSolve* __restrict__ solves, int n_solves, long long n_items,
                     unsigned long long* __restrict__ counter, int* __restrict__ err, PrCtl ctl) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    PrRawRay* bufs = reinterpret_cast<PrRawRay*>(smem) + warp * 2 * kPrStage;
    using WS = WarpSharedT<POL ? 2 : 4, FOLD>;
    WS* wsh = reinterpret_cast<WS*>(smem + kPrWarpsPerCta * 2 * kPrStage * sizeof(PrRawRay)) + warp;
    WarpPipe wp;
    wp.buf[0] = bufs;
    wp.buf[1] = bufs + kPrStage;
    wp.bar[0] = &wsh->bar[0];
    wp.bar[1] = &wsh->bar[1];
    wp.phase = 0;
    if (lane == 0) {
        mbar_init(wp.bar[0], 1);
        mbar_init(wp.bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_proxy_async();
    __syncwarp();
    while (true) {
        long long item = 0;
        if (lane == 0) item = (long long)atomicAdd(counter, 1ull);
        item = __shfl_sync(kFull, item, 0);
        if (item >= n_items) break;
        int lo = 0, hi = n_solves - 1;
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (solves[mid].item_begin <= item) lo = mid;
            else hi = mid - 1;
        }
        const PrSolve& sv = solves[lo];
        const long long local = item - sv.item_begin + sv.item_offset;
        const bool ok = process_item<UNIFORM, FAST, FOLD, POL, LIN>(
            sv, local, wp, *wsh, lane, ctl.wait_limit, item == 0 ? ctl.stall_bytes : 0u);
        if (!ok) {
            if (lane == 0) *static_cast<volatile int*>(err) = 1;
            break;
        }
    }
}

// Dynamic shared memory of a launch: the warps' ray buffers and their state.
constexpr size_t pr_smem_bytes(int variant) {
    const size_t state =
        (variant & 8) ? ((variant & 4) ? sizeof(WarpSharedT<2, true>) : sizeof(WarpSharedT<2, false>))
                      : ((variant & 4) ? sizeof(WarpSharedT<4, true>) : sizeof(WarpSharedT<4, false>));
    return (size_t)kPrWarpsPerCta * (2 * kPrStage * sizeof(PrRawRay) + state);
}

using PrKernel = void (*)(const PrSolve*, int, long long, unsigned long long*, int*, PrCtl);

// Kernel of a variant: bit 0 uniform normal, bit 1 packed sweep, bit 2 folded
// base phase, bit 3 one polarization, bit 4 linear series (PrPlan::variant();
// bit 4 only occurs with bit 1).
template <bool POL>
PrKernel pr_kernel_pol(int v) {
    static const PrKernel table[8] = {
        pr_persistent_kernel<false, false, false, POL, false>,
        pr_persistent_kernel<true, false, false, POL, false>,
        pr_persistent_kernel<false, true, false, POL, false>,
        pr_persistent_kernel<true, true, false, POL, false>,
        pr_persistent_kernel<false, false, true, POL, false>,
        pr_persistent_kernel<true, false, true, POL, false>,
        pr_persistent_kernel<false, true, true, POL, false>,
        pr_persistent_kernel<true, true, true, POL, false>};
    static const PrKernel lin[4] = {  // packed sweeps: uniform x folded
        pr_persistent_kernel<false, true, false, POL, true>,
        pr_persistent_kernel<true, true, false, POL, true>,
        pr_persistent_kernel<false, true, true, POL, true>,
        pr_persistent_kernel<true, true, true, POL, true>};
    if ((v & 16) && (v & 2)) return lin[(v & 1) | ((v >> 1) & 2)];
    return table[v & 7];
}

PrKernel pr_kernel(int variant) {
    return (variant & 8) ? pr_kernel_pol<true>(variant) : pr_kernel_pol<false>(variant);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

struct Arena {
    char* base;
    size_t off = 0;
    template <class T>
    T* take(size_t count) {
        off = align_up(off, 256);
        T* p = reinterpret_cast<T*>(base + off);
        off += count * sizeof(T);
        return p;
    }
};

void normalize3(double v[3]) {
    double n = std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    if (n > 0) {
        v[0] /= n;
        v[1] /= n;
        v[2] /= n;
    }
}

// Range of a world AABB projected on a unit axis through origin o.
void project_box(const double lo[3], const double hi[3], const double o[3], const double ax[3],
                 double* pmin, double* pmax) {
    double mn = INFINITY, mx = -INFINITY;
    for (int c = 0; c < 8; ++c) {
        double p[3] = {(c & 1) ? hi[0] : lo[0], (c & 2) ? hi[1] : lo[1], (c & 4) ? hi[2] : lo[2]};
        double d = (p[0] - o[0]) * ax[0] + (p[1] - o[1]) * ax[1] + (p[2] - o[2]) * ax[2];
        mn = std::min(mn, d);
        mx = std::max(mx, d);
    }
    *pmin = mn;
    *pmax = mx;
}

double box_distance(const double alo[3], const double ahi[3], const double blo[3],
                    const double bhi[3]) {
    double s = 0;
    for (int a = 0; a < 3; ++a) {
        double gap = std::max(0.0, std::max(blo[a] - ahi[a], alo[a] - bhi[a]));
        s += gap * gap;
    }
    return std::sqrt(s);
}

// Upper bound of |k Delta| for chunk radius b, tile radius a, distance d.
double phase_bound(double k, double a, double b, double d) {
    double den = d - 2.0 * b;
    if (den <= 0) return INFINITY;
    return k * (b * b + 2.0 * a * b) / (2.0 * den);
}

// Ray cells of their own length along the beam. The bound above takes tiles and
// cells as balls, but lengths along the line of sight hardly enter the
// residual phase: with A and B the extents across u (for a tile and a cell that
// reach a and b along u0, u within the angle g of u0, A = a_across + a g, B =
// b_across + b g) and v.rho = q_perp.rho_perp + O(|q_perp|^2 / |q|) (u.rho),
//     |k Delta| <= k (B^2 + 2 A B + 2 A^2 b / d) / (2 (d - 2 (B + b))).
// On a mirror lit at grazing incidence, 60 mm along the beam and 1 mm across,
// the ball bound leaves about one ray per cell.
struct DepthCells {
    double cell[3];
    long long n[3];
    double bound, rcp;
};

// Residual phase bounds [rad] such cells are sized for. The ball bound kept the
// true phases of these solves, and so their errors, below what the budget
// allows; these bounds keep the errors near that. Deep tiles: 6 rad in the
// mean tile, 60 in the widest: ten pairs of mirrors, 4 to 19 keV and 3 to 8.5 m apart,
// take 0.08 to 0.6 of the ball bound's time at 3.3e-7 to 4.7e-7 instead of 2.7e-7 to
// 3.0e-7 (6e4 rays x 5e4 points at 3 m: 35.8 ms and 2.7e-7 with the ball bound, 10.0 ms
// and 3.3e-7 so). Flat tiles: a share of the budget.
constexpr double kDeepTileBudget = 6.0, kDeepWideBudget = 60.0;
constexpr double kDepthShare = 0.3;

// Fills `c` and returns true where such cells are clearly fewer than the n[]
// cells of the ball bound. `a_across`, `a_mean`: largest and mean extent of
// the tiles across u0, `a_along`: largest along it, `a_max`: largest radius.
bool depth_cells(double k, double d, double g, double a_across, double a_mean, double a_along,
                 double a_max, const double ext[3], double budget, double tolerance,
                 const long long n[3], DepthCells* c) {
    const double wide = a_across + a_along * g, mean = a_mean + a_along * g;
    const bool deep = a_max > 1.25 * wide;
    // Along the beam: the linear series' argument (b / d)^2 budget within a
    // tenth of the tolerance, with a margin.
    const double b_most = 0.9 * d * std::sqrt(0.1 * tolerance / budget);
    auto eval = [&](double h) -> double {  // <= 1: fits
        double sq = 0.0;
        for (int ax = 0; ax < 2; ++ax) {
            c->cell[ax] = std::min(ext[ax], h);
            sq += 0.25 * c->cell[ax] * c->cell[ax];
        }
        const double across = std::sqrt(sq);
        // At least half of b_most stays for the length along the beam. (Across the
        // whole of it the length came out as zero, which is no cell at all: counted as
        // one, it put rays of any depth into the same chunk.)
        if (!(across * g <= 0.5 * b_most)) return INFINITY;
        const double along =
            std::min(0.5 * ext[2], std::min(b_most - across * g, 0.3 * across / std::max(g, 1e-9)));
        c->cell[2] = 2.0 * along;
        const double b = across + along * g, den = d - 2.0 * (b + along);
        if (!(den > 0.0)) return INFINITY;
        auto bound = [&](double a) {
            return k * (b * b + 2.0 * a * b + 2.0 * a * a * along / d) / (2.0 * den);
        };
        c->rcp = (along + across * g) / std::max(d - along - across, 1e-300);
        c->bound = bound(wide);
        return deep ? std::max(c->bound / std::min(budget, kDeepWideBudget),
                               bound(mean) / kDeepTileBudget)
                    : c->bound / (kDepthShare * budget);
    };
    double lo = 0.0, hi = 2.0 * std::max(ext[0], ext[1]);
    if (!(hi > 0.0)) return false;
    for (int it = 0; it < 100; ++it) {
        const double h = 0.5 * (lo + hi);
        if (eval(h) <= 1.0) lo = h;
        else hi = h;
    }
    if (!(lo > 0.0)) return false;
    eval(lo);
    double cells = 1.0, before = 1.0;
    for (int ax = 0; ax < 3; ++ax) {
        const double cnt = c->cell[ax] > 0 ? std::floor(ext[ax] / c->cell[ax]) + 1.0
                                           : (ext[ax] > 0 ? INFINITY : 1.0);
        if (!(cnt <= 2097151.0)) return false;
        c->n[ax] = (long long)cnt;
        cells *= cnt;
        before *= (double)n[ax];
    }
    return cells < 0.5 * before;
}

// Per-solve planning scratch carved from the arena.
struct SolveBufs {
    double* sum;
    GridProbe* probe;
    double* axes;  // of a rectangular screen (xk_grid.cuh)
    uint64_t *pk_in, *pk_out;
    int *pi_in, *pi_out;
    int* tile_perm;
    double *tpx, *tpy, *tpz, *tile_center;
    double4* rel;
    float* ns;
    unsigned long long* amax;
    uint64_t *rk_in, *rk_out;
    int *ri_in, *ri_out, *flags, *run;
    int* chunk_begin;
    double* chunk_center;
    int* n_chunks;
    int* group_order;
    PrRawRay* recs;
    double* partial;
};

void carve(Arena& a, SolveBufs& b, int n, int m, int n_tiles, int groups, int sum_blocks) {
    const size_t slots = (size_t)n_tiles * kPrTile;
    b.sum = a.take<double>((size_t)(sum_blocks + 1) * kSumFields);
    b.probe = a.take<GridProbe>(1);
    b.axes = a.take<double>(grid_axes_doubles((size_t)m));
    b.pk_in = a.take<uint64_t>(m);
    b.pk_out = a.take<uint64_t>(m);
    b.pi_in = a.take<int>(m);
    b.pi_out = a.take<int>(m);
    b.tile_perm = a.take<int>(slots);
    b.tpx = a.take<double>(slots);
    b.tpy = a.take<double>(slots);
    b.tpz = a.take<double>(slots);
    b.tile_center = a.take<double>(3 * (size_t)n_tiles);
    b.rel = a.take<double4>(slots);
    b.ns = a.take<float>(slots);
    b.amax = a.take<unsigned long long>(4);
    b.rk_in = a.take<uint64_t>(n);
    b.rk_out = a.take<uint64_t>(n);
    b.ri_in = a.take<int>(n);
    b.ri_out = a.take<int>(n);
    b.flags = a.take<int>(n);
    b.run = a.take<int>(n);
    b.chunk_begin = a.take<int>((size_t)n + 1);
    b.chunk_center = a.take<double>(3 * (size_t)n);
    b.n_chunks = a.take<int>(1);
    b.group_order = a.take<int>(groups);
    b.recs = a.take<PrRawRay>(n);
    b.partial = a.take<double>((size_t)groups * 4 * slots);
}

struct HostSolveInfo {
    double f[kSumFields];
    double k = 0, d_lo = 0, quantum = 0, rc[3], pc[3], rlo[3], rhi[3], plo[3], phi[3];
    Frame fr{};
};

// Pinned host area layout: [per-solve summaries][per-solve screen probes][per-solve amax][per-solve
// n_chunks][error word][solve tables].
struct HostLayout {
    size_t sum_off, probe_off, amax_off, nch_off, err_off, tab_off, total;
};

HostLayout host_layout(int count) {
    HostLayout L;
    size_t off = 0;
    L.sum_off = off;
    off = align_up(off + (size_t)count * kSumFields * sizeof(double), 256);
    L.probe_off = off;
    off = align_up(off + (size_t)count * sizeof(GridProbe), 256);
    L.amax_off = off;
    off = align_up(off + 4 * (size_t)count * sizeof(double), 256);
    L.nch_off = off;
    off = align_up(off + (size_t)count * sizeof(int), 256);
    L.err_off = off;
    off = align_up(off + 64, 256);
    L.tab_off = off;
    off = align_up(off + (size_t)count * sizeof(PrSolve), 256);
    L.total = off;
    return L;
}

// Whether a solve's screen is looked at for the tensor-core product
// (xk_grid.cuh): not where the caller set this kernel's own knobs, nor where the
// requested error is near the product's (up to 6e-6; 165 rad of budget stand
// for a tolerance of 6e-5).
bool grid_candidate(const PrOptions& o, size_t n, size_t m) {
    return o.grid && o.sweep < 0 && o.groups == 0 && effective_phase_budget(o) >= 165.0 &&
           n >= kGridMinRays && m >= kGridMinPoints;
}

// Largest residual phase of a pair [rad]: the caller's budget, and B with
// B^2 / (2 k d) = tolerance / 2 (the term left out of the reciprocal). The second
// is the smaller one only where k d is below 8e8 at the default settings, 15 mm at
// 10 keV: 1 mm behind an aperture the budget alone left 1.3e-4 of the field.
double pair_budget(const PrOptions& o, double k, double d) {
    return std::min(effective_phase_budget(o), std::sqrt(o.tolerance * k * d));
}

// Blocks of a solve's summary: at least four elements per thread, because below
// that the reduction of the fields and the host's pass over the blocks' results
// cost more than reading the inputs (10^4 rays: 18 us and 95 KB with 296
// blocks).
int sum_parts(size_t n, size_t m, int sum_blocks) {
    return (int)std::min<size_t>(sum_blocks, std::max<size_t>(1, (std::max(n, m) + 1023) / 1024));
}

int sum_blocks_for(int num_sms) { return std::min(512, std::max(1, 2 * num_sms)); }

// Items per resident warp: the caller's or an autotuned setting.
long long items_per_warp(int n, int m, const PrOptions& opt) {
    long long ipw = opt.items_per_warp;
    if (opt.tune && opt.tune->use) opt.tune->find_ipw((size_t)n, (size_t)m, &ipw);
    return ipw;
}

// Ray groups per tile: enough items to keep every resident warp busy, at
// least four stages of rays per item, partial slots within 1 GiB.
int plan_groups_large(int n, int m, int n_tiles, int num_sms, const PrOptions& opt) {
    if (opt.groups > 0) return std::min(opt.groups, kMaxGroups);
    long long want = (long long)num_sms * 12 * items_per_warp(n, m, opt);
    int g = (int)std::max<long long>(1, (want + n_tiles - 1) / n_tiles);
    g = std::min(g, std::max(1, n / (4 * kPrStage)));
    long long cap = (1LL << 30) / (32LL * n_tiles * kPrTile);
    g = (int)std::max<long long>(1, std::min<long long>(g, cap));
    return std::min(g, kMaxGroups);
}

// The same, and where that leaves less than four items per resident warp (a
// line of 256 points is one tile: 44 items on 1776 warps with 10^4 rays), the
// count that minimises rounds of items x (rays per item + the item's fixed
// cost), items as small as kPrMinItem rays. A number of items per warp that is not the
// default stands as it is.
int plan_groups(int n, int m, int n_tiles, int num_sms, const PrOptions& opt) {
    const int base = plan_groups_large(n, m, n_tiles, num_sms, opt);
    const long long warps = (long long)num_sms * 12;
    if (opt.groups > 0 || items_per_warp(n, m, opt) != PrOptions{}.items_per_warp ||
        (long long)base * n_tiles >= 4 * warps)
        return base;
    constexpr double kItemCost = 60.0;  // set-up, flush and pipeline fill of an item, in rays
    const long long cap = (1LL << 30) / (32LL * n_tiles * kPrTile);
    const int most = (int)std::min<long long>(std::min(n / kPrMinItem, kMaxGroups), cap);
    int best = base;
    double best_cost = 1e300;
    for (int waves = 1; waves <= 8; ++waves)
        for (int g : {(int)std::min<long long>(waves * warps / n_tiles, most), base}) {
            if (g < 1) continue;
            const long long rounds = ((long long)g * n_tiles + warps - 1) / warps;
            const double cost = rounds * ((double)n / g + kItemCost);
            if (cost < best_cost) {
                best_cost = cost;
                best = g;
            }
        }
    return best;
}

}  // namespace

uint32_t PrTuneCache::size_key(size_t n, size_t m) {
    const int nb = n ? std::ilogb((double)n) : 0, mb = m ? std::ilogb((double)m) : 0;
    return (uint32_t)(nb & 0xff) << 8 | (uint32_t)(mb & 0xff);
}

uint64_t PrTuneCache::full_key(double energy_ev, double dist_mm, size_t n, size_t m) {
    const int eb = energy_ev > 0 ? (int)std::lround(std::log2(energy_ev)) : 0;
    const int db = dist_mm > 0 ? (int)std::lround(std::log2(dist_mm)) : 0;
    return (uint64_t)((eb + 128) & 0xff) << 24 | (uint64_t)((db + 128) & 0xff) << 16 |
           size_key(n, m);
}

void PrTuneCache::store(double energy_ev, double dist_mm, size_t n, size_t m, const PrTuned& t) {
    std::lock_guard<std::mutex> lock(mu);
    full[full_key(energy_ev, dist_mm, n, m)] = t;
    ipw[size_key(n, m)] = t.items_per_warp;
}

bool PrTuneCache::find(double energy_ev, double dist_mm, size_t n, size_t m, PrTuned* t) {
    std::lock_guard<std::mutex> lock(mu);
    auto it = full.find(full_key(energy_ev, dist_mm, n, m));
    if (it == full.end()) return false;
    *t = it->second;
    return true;
}

bool PrTuneCache::find_ipw(size_t n, size_t m, long long* ipw_out) {
    std::lock_guard<std::mutex> lock(mu);
    auto it = ipw.find(size_key(n, m));
    if (it == ipw.end()) return false;
    *ipw_out = it->second;
    return true;
}

size_t PrTuneCache::size() {
    std::lock_guard<std::mutex> lock(mu);
    return full.size();
}

void PrTuneCache::clear() {
    std::lock_guard<std::mutex> lock(mu);
    full.clear();
    ipw.clear();
}

const char* const kRouteReasons[kRouteReasonCount] = {
    "",
    "no rays",
    "rays of different energies",
    "non-positive energy",
    "ray and screen bounding boxes overlap",
    "no cell size meets the phase budget",
    "ray cell grid too fine",
    "non-finite ray or screen values",
    "amplitudes outside the FP32 range of the phase-reduced sums"};

Status PrWorkspace::ensure_host(size_t bytes) {
    if (bytes <= host_bytes) return Status::Ok();
    if (host_borrowed) return Status::Err(XK_ERR_OOM, "borrowed pinned area too small");
    if (host) cudaFreeHost(host);
    host = nullptr;
    host_bytes = 0;
    host_err = nullptr;
    XK_CUDA_TRY(cudaMallocHost(&host, bytes));
    host_bytes = bytes;
    return Status::Ok();
}

Status PrWorkspace::ensure_tickets(int count, cudaStream_t stream) {
    const size_t had = tickets.bytes;
    XK_TRY(tickets.ensure(std::max(count, 1) * 4 * sizeof(unsigned)));
    if (tickets.bytes != had) XK_CUDA_TRY(cudaMemsetAsync(tickets.ptr, 0, tickets.bytes, stream));
    return Status::Ok();
}

void PrWorkspace::release() {
    tickets.release();
    arena.release();
    cub_tmp.release();
    solves.release();
    ctrl.release();
    grid.recs.release();
    grid.partial.release();
    for (auto& e : ev)
        if (e) cudaEventDestroy(e);
    ev[0] = ev[1] = nullptr;
    if (host && !host_borrowed) cudaFreeHost(host);
    host = nullptr;
    host_bytes = 0;
    host_err = nullptr;
    host_borrowed = false;
}

size_t pr_plan_bytes(size_t n, size_t m, int num_sms, const PrOptions& opt) {
    if (n == 0 || m == 0) return 0;
    const int sum_blocks = sum_blocks_for(num_sms);
    const int n_tiles = (int)((m + kPrTile - 1) / kPrTile);
    const int g = plan_groups((int)n, (int)m, n_tiles, num_sms, opt);
    Arena a{nullptr, 0};
    SolveBufs b;
    carve(a, b, (int)n, (int)m, n_tiles, g, sum_blocks);
    // CUB radix sort of 64-bit keys + 32-bit values and the scan need at most
    // a few bytes per item; 16 per item plus 1 MiB bounds them.
    return a.off + 16 * std::max(n, m) + (1u << 20) + (2u << 20);
}

namespace {

// Plans the solve as a tensor-core product if its screen and ranges allow.
Status try_grid(const PrSolveIn& in, const GridProbe& probe, const HostSolveInfo& I,
                const PrOptions& opt, const SolveBufs& B, int num_sms, cudaStream_t stream,
                PrPlan* P, int* kernels) {
    PrOptions o = opt;
    bool tuned = false;
    if (opt.tune && opt.tune->use) {
        PrTuned t;
        if (opt.tune->find(P->energy_ev, P->dist_mm, in.n, in.m, &t)) {
            o.phase_budget = std::min(t.phase_budget, opt.phase_budget);
            o.sweep = t.sweep;
            tuned = true;
        }
    }
    if (!grid_candidate(o, in.n, in.m)) return Status::Ok();
    const double* f = I.f;
    GridRanges r{};
    double off2 = 0.0;
    for (int a = 0; a < 3; ++a) {
        r.rlo[a] = I.rlo[a];
        r.rhi[a] = I.rhi[a];
        r.plo[a] = I.plo[a];
        r.phi[a] = I.phi[a];
        r.nlo[a] = f[11 + a];
        r.nhi[a] = f[14 + a];
        r.rc[a] = I.rc[a];
        r.pc[a] = I.pc[a];
        off2 += (I.rc[a] - f[37 + a]) * (I.rc[a] - f[37 + a]);
    }
    r.spread2 = std::max(0.0, f[36] / (double)in.n - off2);
    r.nl_lo = f[34];
    r.nl_hi = f[35];
    const int first = P->one_pol && P->dev.amp_src ? 1 : 0;  // amplitude column summed first
    r.max_amp[0] = first ? f[40] : f[32];
    r.max_amp[1] = P->one_pol ? 0.0 : f[40];
    r.k = I.k;
    GridPlan& g = P->grid_plan;
    if (!grid_plan(probe, r, in.n, in.m, P->one_pol ? 1 : 2, o.tolerance, num_sms, &g))
        return Status::Ok();
    g.rays = in.rays;
    g.pix = in.pix;
    g.out = in.out;
    const double* amps[2][2] = {{in.rays.es_re, in.rays.es_im}, {in.rays.ep_re, in.rays.ep_im}};
    for (int c = 0; c < g.columns; ++c)
        for (int k = 0; k < 2; ++k) g.amps[c][k] = amps[first + c][k];
    for (int k = 0; k < 2; ++k) {
        g.pes[k] = P->pol_es[k];
        g.pep[k] = P->pol_ep[k];
    }
    g.axes = B.axes;
    XK_TRY(grid_axes_enqueue(g, stream));
    ++*kernels;
    P->grid = true;
    P->tuned = tuned;
    P->fast = P->lin = P->fold = false;
    P->n_tiles = g.m_tiles * g.n_tiles;
    P->groups = g.splits;
    P->n_chunks = g.ray_blocks;
    P->phase_bound = 3.14159265358979323846;
    return Status::Ok();
}

// Gives the planned products their scratch, at once and at its largest: growing it solve
// by solve mapped new memory each time (planning a process's first batch of 64 uneven
// solves took 0.27 s, 0.05 so). Where the device has no room for it they run on the
// general kernel, whose scratch is there already.
Status reserve_grids(std::vector<PrPlan>& plans, GridWorkspace& ws) {
    size_t recs = 0, partial = 0;
    for (const PrPlan& P : plans)
        if (!P.routed && P.grid) grid_sizes(P.grid_plan, &recs, &partial);
    Status st = grid_reserve(recs, partial, ws);
    if (st.code != XK_ERR_OOM) return st;
    cudaGetLastError();
    ws.recs.release();
    ws.partial.release();
    for (PrPlan& P : plans) P.grid = P.tuned = false;
    return Status::Ok();
}

}  // namespace

Status pr_plan(const PrSolveIn* in, int count, PrWorkspace& ws, cudaStream_t stream, int num_sms,
               const PrOptions& opt, std::vector<PrPlan>& plans, int* kernels,
               DevBuf* const* arenas) {
    plans.assign(count, PrPlan());
    int nk = 0;
    const int sum_blocks = sum_blocks_for(num_sms);
    std::vector<int> n_tiles(count, 0), groups(count, 0);
    size_t cub_need = 0;
    size_t need = 0;
    for (int s = 0; s < count; ++s) {
        PrPlan& P = plans[s];
        P.out = in[s].out;
        P.m = (int)in[s].m;
        if (in[s].n == 0 || in[s].m == 0) {
            P.routed = true;
            P.route_reason = 1;
            continue;
        }
        if (in[s].n > (size_t)INT32_MAX / 2 || in[s].m > (size_t)INT32_MAX / 2)
            return Status::Err(XK_ERR_INVALID, "too many rays or screen points for one solve");
        const int n = (int)in[s].n, m = (int)in[s].m;
        n_tiles[s] = (m + kPrTile - 1) / kPrTile;
        const int g = plan_groups(n, m, n_tiles[s], num_sms, opt);
        groups[s] = g;
        size_t c1 = 0, c2 = 0, c3 = 0;
        XK_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, c1, (uint64_t*)nullptr,
                                                    (uint64_t*)nullptr, (int*)nullptr,
                                                    (int*)nullptr, n));
        XK_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, c2, (uint64_t*)nullptr,
                                                    (uint64_t*)nullptr, (int*)nullptr,
                                                    (int*)nullptr, m));
        XK_CUDA_TRY(cub::DeviceScan::InclusiveSum(nullptr, c3, (int*)nullptr, (int*)nullptr, n));
        cub_need = std::max(cub_need, std::max(c1, std::max(c2, c3)));
        Arena a{nullptr, arenas ? 0 : need};
        SolveBufs b;
        carve(a, b, n, m, n_tiles[s], g, sum_blocks);
        if (arenas) XK_TRY(arenas[s]->ensure(a.off + 256));
        else need = a.off;
    }
    XK_TRY(ws.cub_tmp.ensure(cub_need + 256));
    if (!arenas) {
        Status st = ws.arena.ensure(need + 256);
        if (st.code == XK_ERR_OOM && ws.grid.recs.bytes) {
            // Earlier products' scratch is in the way.
            cudaGetLastError();
            ws.grid.recs.release();
            ws.grid.partial.release();
            st = ws.arena.ensure(need + 256);
        }
        XK_TRY(st);
    }
    const HostLayout HL = host_layout(count);
    XK_TRY(ws.ensure_host(HL.total));
    char* hbase = static_cast<char*>(ws.host);
    double* h_sum = reinterpret_cast<double*>(hbase + HL.sum_off);
    GridProbe* h_probe = reinterpret_cast<GridProbe*>(hbase + HL.probe_off);
    double* h_amax = reinterpret_cast<double*>(hbase + HL.amax_off);
    int* h_nch = reinterpret_cast<int*>(hbase + HL.nch_off);
    XK_TRY(ws.ensure_tickets(count, stream));
    unsigned* tickets = ws.tickets.as<unsigned>();

    std::vector<SolveBufs> bufs(count);
    {
        size_t off = 0;
        for (int s = 0; s < count; ++s) {
            if (plans[s].routed) continue;
            Arena a{arenas ? arenas[s]->as<char>() : ws.arena.as<char>(), arenas ? 0 : off};
            carve(a, bufs[s], (int)in[s].n, (int)in[s].m, n_tiles[s], groups[s], sum_blocks);
            off = a.off;
        }
    }

    // --- A. summaries ------------------------------------------------------
    bool any = false;
    std::vector<SummaryArgs> sums;
    std::vector<ProbeArgs> probes;
    for (int s = 0; s < count; ++s) {
        if (plans[s].routed) continue;
        any = true;
        const int parts = sum_parts(in[s].n, in[s].m, sum_blocks);
        sums.push_back({in[s].rays, in[s].pix, (int)in[s].n, (int)in[s].m, 0, parts, bufs[s].sum,
                        bufs[s].probe, tickets + 4 * s, h_sum + s * kSumFields});
        if (grid_candidate(opt, in[s].n, in[s].m)) {
            h_probe[s] = GridProbe{};
            probes.push_back({in[s].pix, (int)in[s].m, 0, 0, bufs[s].sum + parts * kSumFields + 33,
                              bufs[s].probe, tickets + 4 * s + 1, h_probe + s});
        }
    }
    if (sums.size() == 1)
        XK_TRY((launch_solves<1, SummaryBatch<1>>(summary_kernel<1>, sums, stream, &nk)));
    else
        XK_TRY((launch_solves<kSolvesPerLaunch, SummaryBatch<kSolvesPerLaunch>>(
            summary_kernel<kSolvesPerLaunch>, sums, stream, &nk)));
    XK_TRY(grid_probe_enqueue(probes, stream, &nk));
    if (!any) {
        if (kernels) *kernels += nk;
        return Status::Ok();
    }
    XK_CUDA_TRY(cudaStreamSynchronize(stream));

    std::vector<HostSolveInfo> info(count);
    for (int s = 0; s < count; ++s) {
        PrPlan& P = plans[s];
        if (P.routed) continue;
        HostSolveInfo& I = info[s];
        std::memcpy(I.f, h_sum + s * kSumFields, sizeof(I.f));
        const double* f = I.f;
        if (!(f[26] == 0.0)) {
            // NaN or infinite inputs: the FP64 sum propagates them the way
            // diffraction.rs:67-117 does; the planner's geometry would not.
            P.routed = true;
            P.route_reason = 7;
            continue;
        }
        const double most = std::max(f[32], f[40]);
        if (most > kF32AmpMax || (most > 0.0 && most < kF32AmpMin)) {
            P.routed = true;
            P.route_reason = 8;
            continue;
        }
        if (!(f[9] == f[10])) {
            P.routed = true;
            P.route_reason = 2;
            continue;
        }
        I.k = (f[9] / kChbar) * 1e7;
        if (!(I.k > 0) || !std::isfinite(I.k)) {
            P.routed = true;
            P.route_reason = 3;
            continue;
        }
        P.uniform_normal = f[11] == f[14] && f[12] == f[15] && f[13] == f[16];
        // One common polarization (es_j, ep_j) ~ (es_0, ep_0): sum A over
        // a_j = es_j, Ep = (ep_0 / es_0) A; with es_0 = 0 every es_j is 0 and
        // a_j = ep_j.
        const double a0r = f[28], a0i = f[29], b0r = f[30], b0i = f[31];
        const bool es0 = a0r != 0.0 || a0i != 0.0, ep0 = b0r != 0.0 || b0i != 0.0;
        P.one_pol = opt.polarization != 0 && f[27] <= kOnePolTol && (es0 || ep0);
        if (P.one_pol && es0) {
            // ep_0 / es_0 in extended precision (|es_0|^2 cannot underflow);
            // a ratio beyond FP64's range keeps both columns.
            const long double ar = a0r, ai = a0i, br = b0r, bi = b0i;
            const long double d = ar * ar + ai * ai;
            const double pr = (double)((br * ar + bi * ai) / d);
            const double pi = (double)((bi * ar - br * ai) / d);
            if (std::isfinite(pr) && std::isfinite(pi)) {
                P.dev.amp_src = 0;
                P.pol_es[0] = 1.0;
                P.pol_es[1] = 0.0;
                P.pol_ep[0] = pr;
                P.pol_ep[1] = pi;
            } else {
                P.one_pol = false;
            }
        } else if (P.one_pol) {
            P.dev.amp_src = 1;
            P.pol_es[0] = P.pol_es[1] = 0.0;
            P.pol_ep[0] = 1.0;
            P.pol_ep[1] = 0.0;
        }
        for (int a = 0; a < 3; ++a) {
            I.rlo[a] = f[3 + a];
            I.rhi[a] = f[6 + a];
            I.plo[a] = f[20 + a];
            I.phi[a] = f[23 + a];
            I.rc[a] = f[a] / (double)in[s].n;
            I.pc[a] = f[17 + a] / (double)in[s].m;
        }
        I.d_lo = box_distance(I.rlo, I.rhi, I.plo, I.phi);
        {
            // 2^E bounds every screen and ray coordinate; multiples of 2^(E-52)
            // then subtract from any screen coordinate exactly.
            double amax = 0.0;
            for (int a = 0; a < 3; ++a)
                amax = std::max(amax, std::max(std::max(std::fabs(I.plo[a]), std::fabs(I.phi[a])),
                                               std::max(std::fabs(I.rlo[a]), std::fabs(I.rhi[a]))));
            const int e = amax > 0 ? std::ilogb(amax) + 2 : -960;
            I.quantum = std::ldexp(1.0, e - 52);
        }
        P.energy_ev = f[9];
        P.dist_mm = std::sqrt((I.pc[0] - I.rc[0]) * (I.pc[0] - I.rc[0]) +
                              (I.pc[1] - I.rc[1]) * (I.pc[1] - I.rc[1]) +
                              (I.pc[2] - I.rc[2]) * (I.pc[2] - I.rc[2]));
        if (!(I.d_lo > 0)) {
            P.routed = true;
            P.route_reason = 4;
            continue;
        }
        double u0[3] = {I.pc[0] - I.rc[0], I.pc[1] - I.rc[1], I.pc[2] - I.rc[2]};
        if (u0[0] * u0[0] + u0[1] * u0[1] + u0[2] * u0[2] == 0) u0[2] = 1;
        normalize3(u0);
        double helper[3] = {std::fabs(u0[0]) < 0.9 ? 1.0 : 0.0, std::fabs(u0[0]) < 0.9 ? 0.0 : 1.0,
                            0.0};
        double dot = helper[0] * u0[0] + helper[1] * u0[1] + helper[2] * u0[2];
        double e1[3] = {helper[0] - dot * u0[0], helper[1] - dot * u0[1], helper[2] - dot * u0[2]};
        normalize3(e1);
        double e2[3] = {u0[1] * e1[2] - u0[2] * e1[1], u0[2] * e1[0] - u0[0] * e1[2],
                        u0[0] * e1[1] - u0[1] * e1[0]};
        for (int i = 0; i < 3; ++i) {
            I.fr.e1[i] = e1[i];
            I.fr.e2[i] = e2[i];
            I.fr.u0[i] = u0[i];
        }
        if (grid_candidate(opt, in[s].n, in[s].m))
            XK_TRY(try_grid(in[s], h_probe[s], I, opt, bufs[s], num_sms, stream, &P, &nk));
    }

    XK_TRY(reserve_grids(plans, ws.grid));

    // --- B. screen tiles ----------------------------------------------------
    any = false;
    for (int s = 0; s < count; ++s) {
        PrPlan& P = plans[s];
        if (P.routed || P.grid) continue;
        any = true;
        HostSolveInfo& I = info[s];
        SolveBufs& B = bufs[s];
        const int m = (int)in[s].m;
        Frame pf = I.fr;
        pf.ox = I.pc[0];
        pf.oy = I.pc[1];
        pf.oz = I.pc[2];
        const double* axes[3] = {I.fr.e1, I.fr.e2, I.fr.u0};
        const double qmax[3] = {65535.0, 65535.0, 2097151.0};
        for (int ax = 0; ax < 3; ++ax) {
            double mn, mx;
            project_box(I.plo, I.phi, I.pc, axes[ax], &mn, &mx);
            pf.lo[ax] = mn;
            pf.scale[ax] = (mx > mn) ? qmax[ax] / (mx - mn) : 0.0;
        }
        // A screen deeper than it is wide, such as a second mirror seen end-on
        // (2 mm wide, 1 um high): one scale for both transverse axes, so that
        // tiles are as wide as they are high. Separate scales made every tile
        // of that mirror fourteen times wider than it need be.
        const double deep = qmax[2] / pf.scale[2], wide = qmax[0] / std::min(pf.scale[0], pf.scale[1]);
        if (pf.scale[0] > 0.0 && pf.scale[1] > 0.0 && pf.scale[2] > 0.0 && deep > wide)
            pf.scale[0] = pf.scale[1] = std::min(pf.scale[0], pf.scale[1]);
        pixel_keys_kernel<<<(m + 255) / 256, 256, 0, stream>>>(in[s].pix, m, pf, B.pk_in, B.pi_in,
                                                                B.amax);
        XK_CUDA_TRY(cudaGetLastError());
        size_t tmp = ws.cub_tmp.bytes;
        // A screen without depth has zeros in the keys' low 21 bits.
        XK_CUDA_TRY(cub::DeviceRadixSort::SortPairs(ws.cub_tmp.ptr, tmp, B.pk_in, B.pk_out, B.pi_in,
                                                    B.pi_out, m, pf.scale[2] > 0.0 ? 0 : 21, 53,
                                                    stream));
        // No tile reaches further than the screen's diagonal, below 2 units of 2^e; 2^22
        // tiles (2^30 points) of 2^41 fit in 64 bits.
        double diag = 0.0;
        for (int a = 0; a < 3; ++a) diag = std::hypot(diag, I.phi[a] - I.plo[a]);
        const double sum_scale = diag > 0.0 ? std::ldexp(1.0, 40 - std::ilogb(diag)) : 1.0;
        tile_kernel<<<(n_tiles[s] * 32 + 255) / 256, 256, 0, stream>>>(
            in[s].pix, m, n_tiles[s], pf, I.quantum, 1.0 / I.quantum, sum_scale,
            make_double3(2.0 * I.f[11], 2.0 * I.f[12], 2.0 * I.f[13]), B.pi_out, B.rel, B.ns,
            B.tile_perm, B.tpx, B.tpy, B.tpz, B.tile_center,
            B.amax, tickets + 4 * s + 2, h_amax + 4 * s);
        XK_CUDA_TRY(cudaGetLastError());
        nk += 2;
    }
    if (any) XK_CUDA_TRY(cudaStreamSynchronize(stream));

    // --- C. ray chunks ------------------------------------------------------
    for (int s = 0; s < count; ++s) {
        PrPlan& P = plans[s];
        if (P.routed || P.grid) continue;
        HostSolveInfo& I = info[s];
        SolveBufs& B = bufs[s];
        const int n = (int)in[s].n;
        const double a_max = h_amax[4 * s] * 1.001;
        const double k = I.k;
        // Autotuned settings of this solve's bucket, if any.
        PrOptions o = opt;
        if (opt.tune && opt.tune->use) {
            PrTuned t;
            if (opt.tune->find(P.energy_ev, P.dist_mm, in[s].n, in[s].m, &t)) {
                o.phase_budget = std::min(t.phase_budget, opt.phase_budget);
                o.sweep = t.sweep;
                P.tuned = true;
            }
        }
        CellGrid cg{};
        cg.fr = I.fr;
        cg.fr.ox = I.rc[0];
        cg.fr.oy = I.rc[1];
        cg.fr.oz = I.rc[2];
        double ext[3];
        const double* axes[3] = {I.fr.e1, I.fr.e2, I.fr.u0};
        for (int ax = 0; ax < 3; ++ax) {
            double mn, mx;
            project_box(I.rlo, I.rhi, I.rc, axes[ax], &mn, &mx);
            cg.fr.lo[ax] = mn;
            ext[ax] = mx - mn;
        }
        auto cell_radius = [&](double h, double cell[3]) {
            double sq = 0;
            for (int ax = 0; ax < 3; ++ax) {
                cell[ax] = ext[ax] <= h ? ext[ax] : h;
                sq += 0.25 * cell[ax] * cell[ax];
            }
            return std::sqrt(sq);
        };
        double cell[3];
        const double budget = pair_budget(o, k, I.d_lo);
        double h_hi = 2.0 * std::max(ext[0], std::max(ext[1], ext[2])) + 1e-300;
        double h_lo = 0.0;
        if (phase_bound(k, a_max, cell_radius(h_hi, cell), I.d_lo) <= budget) {
            h_lo = h_hi;
        } else {
            for (int it = 0; it < 200; ++it) {
                double h = 0.5 * (h_lo + h_hi);
                if (phase_bound(k, a_max, cell_radius(h, cell), I.d_lo) <= budget) h_lo = h;
                else h_hi = h;
            }
        }
        const double h = h_lo;
        const double b_max = cell_radius(h, cell);
        if (!(h > 0)) {
            P.routed = true;
            P.route_reason = 5;
            continue;
        }
        bool too_fine = false;
        for (int ax = 0; ax < 3; ++ax) {
            cg.cell[ax] = cell[ax];
            double cnt = cell[ax] > 0 ? std::floor(ext[ax] / cell[ax]) + 1.0 : 1.0;
            if (cnt > 2097151.0) too_fine = true;
            cg.n[ax] = (long long)cnt;
        }
        if (too_fine) {
            P.routed = true;
            P.route_reason = 6;
            continue;
        }
        cg.quantum = I.quantum;
        cg.inv_quantum = 1.0 / I.quantum;
        P.phase_bound = phase_bound(k, a_max, b_max, I.d_lo);
        // |e| = |u.rho| / |q| <= b / (d_lo - b): the series reciprocal's
        // argument.
        P.rcp_bound = b_max / std::max(I.d_lo - b_max, 1e-300);
        // Largest angle between a ray-to-point line and u0, and longest line.
        double tilt = 0.0, d_hi = 0.0;
        {
            double side2 = 0.0;
            for (int ax = 0; ax < 2; ++ax) {
                double mn, mx;
                project_box(I.plo, I.phi, I.rc, axes[ax], &mn, &mx);
                const double gap = std::max(mx - cg.fr.lo[ax], cg.fr.lo[ax] + ext[ax] - mn);
                side2 += gap * gap;
            }
            tilt = std::sqrt(side2) / I.d_lo;
            for (int a = 0; a < 3; ++a) {
                const double gap = std::max(I.phi[a] - I.rlo[a], I.rhi[a] - I.plo[a]);
                d_hi += gap * gap;
            }
            d_hi = std::sqrt(d_hi);
            DepthCells dc;
            if (depth_cells(k, I.d_lo, tilt, h_amax[4 * s + 1] * 1.001,
                            h_amax[4 * s + 3] / n_tiles[s], h_amax[4 * s + 2] * 1.001, a_max, ext,
                            budget, o.tolerance, cg.n, &dc)) {
                for (int ax = 0; ax < 3; ++ax) {
                    cg.cell[ax] = dc.cell[ax];
                    cg.n[ax] = dc.n[ax];
                }
                P.phase_bound = dc.bound;
                P.rcp_bound = dc.rcp;
            }
        }
        P.fast = o.sweep >= 1 || (o.sweep < 0 && P.rcp_bound <= kSeriesRcpBound);
        // The linear series drops r0 e^2: a relative error of at most e^2 in
        // the reciprocal, |residual phase| e^2 in the phase (a bias shared by
        // all pairs). Used where that stays below a tenth of the tolerance.
        P.lin = P.fast && (o.sweep == 2 ||
                           (o.sweep < 0 &&
                            P.rcp_bound * P.rcp_bound * budget <= 0.1 * o.tolerance));
        {
            // Fold the base phase into the sweep when ray groups span many
            // chunks and chunks hold few rays (near field): per-chunk set-up
            // and flushes then disappear, at the price of a phase add per
            // pair in the sweep. Non-empty cells bound the chunk count from
            // above.
            double cells = 1.0;
            for (int ax = 0; ax < 3; ++ax) cells *= (double)cg.n[ax];
            const double est_chunks = std::min(cells, (double)n);
            const int base = plan_groups_large(n, (int)in[s].m, n_tiles[s], num_sms, opt);
            P.fold = est_chunks >= kFoldChunksPerGroup * (double)base &&
                     (double)n < kFoldRaysPerChunk * est_chunks;
        }

        ray_keys_kernel<<<(n + 255) / 256, 256, 0, stream>>>(in[s].rays, n, cg, B.rk_in, B.ri_in);
        XK_CUDA_TRY(cudaGetLastError());
        size_t tmp = ws.cub_tmp.bytes;
        // Cell indices: as many key bits as there are cells (a sort pass takes
        // eight bits and 9 us however few the rays).
        double cells = 1.0;
        for (int ax = 0; ax < 3; ++ax) cells *= (double)cg.n[ax];
        const int key_bits = std::min(63, std::max(1, std::ilogb(cells) + 1));
        XK_CUDA_TRY(cub::DeviceRadixSort::SortPairs(ws.cub_tmp.ptr, tmp, B.rk_in, B.rk_out, B.ri_in,
                                                    B.ri_out, n, 0, key_bits, stream));
        head_flags_kernel<<<(n + 255) / 256, 256, 0, stream>>>(B.rk_out, n, B.flags);
        XK_CUDA_TRY(cudaGetLastError());
        tmp = ws.cub_tmp.bytes;
        XK_CUDA_TRY(cub::DeviceScan::InclusiveSum(ws.cub_tmp.ptr, tmp, B.flags, B.run, n, stream));
        chunk_table_kernel<<<(n + 255) / 256, 256, 0, stream>>>(B.rk_out, B.flags, B.run, n, cg,
                                                                 B.chunk_begin, B.chunk_center,
                                                                 B.n_chunks, h_nch + s);
        XK_CUDA_TRY(cudaGetLastError());
        records_kernel<<<(n + 255) / 256, 256, 0, stream>>>(in[s].rays, n, B.ri_out, B.run,
                                                             B.chunk_center, B.recs);
        XK_CUDA_TRY(cudaGetLastError());
        nk += 5;
        // Items that all start at once need no order.
        const bool ordered = (long long)groups[s] * n_tiles[s] > (long long)num_sms * 12;
        if (ordered) {
            group_order_kernel<<<1, 1024, 0, stream>>>(B.chunk_begin, B.n_chunks, n, groups[s],
                                                       B.group_order);
            XK_CUDA_TRY(cudaGetLastError());
            ++nk;
        }

        PrSolve& D = P.dev;
        D.recs = B.recs;
        D.chunk_begin = B.chunk_begin;
        D.chunk_center = B.chunk_center;
        D.n_chunks_dev = B.n_chunks;
        D.tpx = B.tpx;
        D.tpy = B.tpy;
        D.tpz = B.tpz;
        D.tile_center = B.tile_center;
        D.tile_rel = B.rel;
        D.tile_ns = B.ns;
        {
            // Flat tiles: the first dropped term of the expansion of |q|,
            // 21/1024 e^6 D, below 1e-8 turn. |e| <= (2 |u.s| + s^2 / D) / D,
            // u.s at most the tile's extent along u0 plus its extent across
            // times the angle between u and u0.
            const double us = h_amax[4 * s + 2] + h_amax[4 * s + 1] * tilt;
            const double e = (2.0 * us + a_max * a_max / I.d_lo) * 1.01 / I.d_lo;
            D.flat = k / 6.28 * d_hi * 0.0206 * std::pow(e, 6.0) < 1e-8;
        }
        D.group_order = ordered ? B.group_order : nullptr;
        D.partial = B.partial;
        D.item_begin = 0;
        D.item_offset = 0;
        D.subs = 1;
        D.n_items = (long long)n_tiles[s] * groups[s];
        D.n_rays = n;
        D.n_tiles = n_tiles[s];
        D.groups = groups[s];
        D.k = k;
        {
            // k/(2 pi) as a double-double, k taken as the FP64 value the
            // reference computes (E / CHBAR * 1e7).
            const long double kt_ld = (long double)k / (2.0L * 3.14159265358979323846264338327950288L);
            D.kt = (double)kt_ld;
            D.kt_lo = (double)(kt_ld - (long double)D.kt);
        }
        D.unx = (float)I.f[11];
        D.uny = (float)I.f[12];
        D.unz = (float)I.f[13];
        P.tile_perm = B.tile_perm;
        P.n_tiles = n_tiles[s];
        P.groups = groups[s];
        P.n_chunks_host = h_nch + s;
    }
    if (kernels) *kernels += nk;
    return Status::Ok();
}

Status pr_zero_partials(const PrPlan& P, cudaStream_t stream) {
    const size_t slots = (size_t)P.n_tiles * kPrTile;
    XK_CUDA_TRY(cudaMemsetAsync(P.dev.partial, 0, (size_t)P.groups * 4 * slots * sizeof(double),
                                stream));
    return Status::Ok();
}

Status pr_launch(const PrSolve* d_table, int n_solves, long long n_items, int variant,
                 unsigned long long* d_counter, int* d_err, cudaStream_t stream, int num_sms,
                 int max_ctas_per_sm, const PrCtl& ctl) {
    if (n_items <= 0) return Status::Ok();
    PrKernel kern = pr_kernel(variant);
    const size_t smem = pr_smem_bytes(variant);
    XK_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    XK_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kPrWarpsPerCta * 32,
                                                              smem));
    per_sm = std::max(per_sm, 1);
    if (max_ctas_per_sm > 0) per_sm = std::min(per_sm, max_ctas_per_sm);
    long long grid = (long long)num_sms * per_sm;
    grid = std::max<long long>(1, std::min(grid, (n_items + kPrWarpsPerCta - 1) / kPrWarpsPerCta));
    kern<<<(unsigned)grid, kPrWarpsPerCta * 32, smem, stream>>>(d_table, n_solves, n_items,
                                                                d_counter, d_err, ctl);
    XK_CUDA_TRY(cudaGetLastError());
    return Status::Ok();
}

Status pr_finalize(const PrPlan& P, cudaStream_t stream) {
    const int slots = P.n_tiles * kPrTile;
    finalize_kernel<<<slots / kFinSlots, kFinSlots * kFinLanes, 0, stream>>>(
        P.dev.partial, P.tile_perm, P.groups, slots, P.out, P.one_pol ? 1 : 0,
        make_double2(P.pol_es[0], P.pol_es[1]), make_double2(P.pol_ep[0], P.pol_ep[1]));
    XK_CUDA_TRY(cudaGetLastError());
    return Status::Ok();
}

Status pr_reserve_plan_host(PrWorkspace& ws, int count, int num_sms) {
    return ws.ensure_host(host_layout(count).total);
}

Status pr_reserve_exec(PrWorkspace& ws, int count, int num_sms) {
    const HostLayout HL = host_layout(count);
    XK_TRY(ws.ensure_host(HL.total));
    XK_TRY(ws.solves.ensure(std::max<size_t>(1, count) * sizeof(PrSolve)));
    XK_TRY(ws.ctrl.ensure(kPrCtrlBytes));
    if (!ws.ev[0]) XK_CUDA_TRY(cudaEventCreate(&ws.ev[0]));
    if (!ws.ev[1]) XK_CUDA_TRY(cudaEventCreate(&ws.ev[1]));
    return Status::Ok();
}

Status pr_execute_enqueue(std::vector<PrPlan>& plans, PrWorkspace& ws, cudaStream_t stream,
                          int num_sms, bool time_kernels, PrExecReport* rep) {
    PrExecReport local;
    PrExecReport& R = rep ? *rep : local;
    const int count = (int)plans.size();
    const HostLayout HL = host_layout(count);
    XK_TRY(pr_reserve_exec(ws, count, num_sms));
    char* hbase = static_cast<char*>(ws.host);
    PrSolve* h_tab = reinterpret_cast<PrSolve*>(hbase + HL.tab_off);
    ws.host_err = reinterpret_cast<int*>(hbase + HL.err_off);
    *ws.host_err = 0;
    unsigned long long* d_counters = reinterpret_cast<unsigned long long*>(ws.ctrl.ptr);

    // Group the planned solves by kernel variant into contiguous tables.
    struct Launch {
        int first, count;
        long long items;
        int variant;
    };
    std::vector<Launch> launches;
    int tab = 0;
    for (int variant = 0; variant < kPrVariants; ++variant) {
        Launch L{tab, 0, 0, variant};
        for (int s = 0; s < count; ++s) {
            PrPlan& P = plans[s];
            if (P.routed || P.grid || P.variant() != variant) continue;
            P.dev.item_begin = L.items;
            h_tab[tab++] = P.dev;
            L.items += P.dev.n_items;
            L.count++;
            XK_TRY(pr_zero_partials(P, stream));
        }
        if (L.count) launches.push_back(L);
    }
    bool any_grid = false;
    for (const PrPlan& P : plans) any_grid |= !P.routed && P.grid;
    if (tab == 0 && !any_grid) return Status::Ok();
    if (tab) {
        XK_CUDA_TRY(cudaMemsetAsync(ws.ctrl.ptr, 0, kPrCtrlBytes, stream));
        XK_CUDA_TRY(cudaMemcpyAsync(ws.solves.ptr, h_tab, (size_t)tab * sizeof(PrSolve),
                                    cudaMemcpyHostToDevice, stream));
    }
    if (time_kernels) XK_CUDA_TRY(cudaEventRecord(ws.ev[0], stream));
    int li = 0;
    PrCtl ctl = ws.ctl;
    ws.ctl.stall_bytes = 0;  // the stall test hook arms one execution only
    for (const Launch& L : launches) {
        XK_TRY(pr_launch(reinterpret_cast<const PrSolve*>(ws.solves.ptr) + L.first, L.count,
                         L.items, L.variant, d_counters + li, ws.host_err, stream, num_sms, 0, ctl));
        ctl.stall_bytes = 0;
        R.kernels += 1;
        R.n_items += L.items;
        ++li;
    }
    for (const PrPlan& P : plans) {
        if (P.routed || !P.grid) continue;
        XK_TRY(grid_enqueue(P.grid_plan, ws.grid, ws.host_err, ctl.wait_limit, ctl.stall_bytes != 0,
                            stream, &R.kernels));
        ctl.stall_bytes = 0;
        R.n_items += (long long)P.n_tiles * P.groups;
    }
    if (time_kernels) XK_CUDA_TRY(cudaEventRecord(ws.ev[1], stream));
    for (int s = 0; s < count; ++s) {
        PrPlan& P = plans[s];
        if (P.routed || P.grid) continue;
        XK_TRY(pr_finalize(P, stream));
        R.kernels += 1;
    }
    return Status::Ok();
}

Status pr_execute_finish(std::vector<PrPlan>& plans, PrWorkspace& ws, PrExecReport* rep) {
    if (rep && rep->kernels > 0 && ws.ev[0]) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, ws.ev[0], ws.ev[1]) == cudaSuccess) rep->main_kernel_ms = ms;
    }
    for (auto& P : plans)
        if (!P.routed && !P.grid && P.n_chunks_host) P.n_chunks = *P.n_chunks_host;
    if (ws.host_err && *ws.host_err != 0)
        return Status::Err(XK_ERR_TIMEOUT, "phase-reduced kernel: a bounded wait for a ray stage ran out");
    return Status::Ok();
}

}  // namespace xk
