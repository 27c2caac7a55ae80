// Phase-reduced Kirchhoff sum on a rectangular screen as a tensor-core product.
//
// On a screen whose points are (a_i, b_l, c) the squared distance to a ray is a
// sum of a row part and a column part, and only the square root couples them.
// For a tile with reference point p0 = (a0, b0, c), u = a_i - a0, v = b_l - b0,
// A = a0 - r_a, B = b0 - r_b, D = |p0 - r|:
//     |p - r|^2 = D^2 + dS + dT,  dS = u (u + 2A),  dT = v (v + 2B),
//     |p - r|   = D + (sqrt(D^2 + dS) - D) + (sqrt(D^2 + dT) - D) + E/k,
//     E         = -k dS dT / (4 D^3) (1 + O((dS + dT) / D^2)).
// The first three terms make a phase that is a row phase plus a column phase,
// so the tile is a complex matrix product over the rays, and
// exp(i E) = 1 + i E - E^2 / 2 + O(E^3) adds one or two more products with the same
// ray index as contraction, because E is a row factor dS times a column factor dT.
// The planner takes the product only where the dropped terms stay far below the
// requested tolerance (grid_plan). The amplitude (nl + n.(p - r)/|p - r|) /
// |p - r| varies along a tile by 1e-7 to 1e-2; its ray part at p0 goes to the
// columns, its first-order change to each side as a factor.
//
//   * grid_records_kernel: per (tile, ray) 64 bytes: k D in turns, reduced in
//     double-double (k D reaches 1e12 rad), the linear phase coefficients as
//     hi + lo floats, the amplitude at p0.
//   * grid_product_kernel: CTA pairs (tcgen05 cta_group::2, 256 rows x 128 or
//     256 columns), the structure of fresnel_pair_kernel: producer warps turn rays
//     into f16 hi + lo phasor tiles in shared memory, one thread issues
//     A_hi B_hi + A_hi B_lo + A_lo B_hi + A_1 B_1 per block of 32 rays, four
//     epilogue warps drain the f32 accumulator every `seg` blocks.
//   * grid_reduce_kernel: adds the ray splits in FP64, in split order, applies
//     i k / (4 pi) and the polarization.
//
// Row and column phases are evaluated as in the Fresnel product: sqrt(D^2 + dS)
// - D = dS / (2D) - dS^2 / (8 D^3), where dS / (2D) = u^2 h + u (2 h A), h =
// 1 / (2D): u^2 h0 is reduced in FP64 per row, u (2 h A) is an exact FP32
// product of hi + lo parts, u^2 (h - h0) and the second-order term are small.

#include <algorithm>
#include <cmath>
#include <cstring>

#include "xk_dd.cuh"
#include "xk_grid.cuh"
#include "xk_phasor.cuh"

namespace xk {
namespace {

using namespace phasor;

constexpr int kTileM = 256;
constexpr uint32_t kGA = 128 * 128;  // 128 rows x 128 B: one f16 tile of a CTA
constexpr uint32_t kGTiles = 12 * kGA;  // the stages' tiles, in every form
constexpr uint32_t kGRays = 3 * kFRays * 64;  // staged ray records
constexpr int kGEpiBufs = 3;  // staging buffers per epilogue warp
constexpr uint32_t kDrainBytes = 32 * 16 * 4;  // 32 rows x 16 columns of a partial
constexpr size_t kGSmem = 1024 + kGTiles + kGRays + 4 * kGEpiBufs * kDrainBytes + 256;
static_assert(kGSmem <= 227 * 1024, "shared memory");

// The product's three forms. The first two have two stages of 32 rays, each of six
// tiles: hi, lo and first order of A (128 rows) and of B (128 rows).
// Narrow: 128 columns per tile. A row of either operand holds its rays' (re, im)
// words, and B has a real-part and an imaginary-part row per column; the two
// accumulators of 256 TMEM columns alternate between segments.
// Wide: 256 columns. A row holds 32 real parts, then 32 imaginary parts, so that
// one B row per column serves both parts of the field (Ar Br - Ai Bi and Ar Bi +
// Ai Br, the sign a bit of the instruction): half the phasor stores per column,
// and the A phasors serve twice the columns. One accumulator each for the real
// and the imaginary part; a part is drained while the other's products run.
// 2^20 rays x 512^2 points: 7.5 ms narrow, 6.3 ms wide (first calls; 8.5 and
// 7.1 ms in a row, the chip at its power limit and 1.55 GHz). In the wide form
// the tensor pipe is busy 72 % of the time (narrow 43 %) and shared memory 75 %
// (products 35, record loads 22, stores 18 %).
// Second: the wide form with the product A_2 B_2 of the second order, X dS^2 times
// -W (4 pi q dT)^2 / 2, in three stages of 16 rays: a row of a tile holds 16 real and 16
// imaginary hi parts, then the lo parts; of another, first, then second orders. For the
// screens on which E is past first order on whole tiles. 20 MMAs per accumulator and 32
// rays instead of 16: 8.7 ms on 2^20 rays x 512^2 points at 0.5 m, where the wide form
// would take 7.1. First order alone, on tiles small enough for it, took 4.0 and 7.9 ms on
// 2^18 rays x 256^2 points +-1 mm at 1 m, 10 and 20 keV; so 1.07 and 3.6.
template <int FORM>
struct Form {
    static constexpr bool kWide = FORM != kFormNarrow, kSecond = FORM == kFormSecond;
    static constexpr int kTileN = kWide ? 256 : 128;
    static constexpr int kAcc = kWide ? 2 : 1;  // accumulators of a segment
    static constexpr int kProdWarps = kWide ? 8 : 12;
    static constexpr int kThreads = 32 + kFEpiThreads + 32 * kProdWarps + 32;
    static constexpr int kRays = kSecond ? 16 : kFRays;  // of a stage
    static constexpr int kStages = kSecond ? 3 : 2;
    static constexpr int kRayBufs = kSecond ? 6 : 3;
    static constexpr uint32_t kStage = kGTiles / kStages, kRayBytes = kRays * 64;
    static_assert(kRayBufs * kRayBytes == kGRays, "ray buffers");
};
constexpr double kGridShare = 0.1;  // of the tolerance: the dropped orders of exp(iE)
constexpr double kGridMostE = 300.0;  // largest E per tolerance
constexpr double kSecondCost = 1.1;   // of the narrow form's time per padded pair
constexpr double kGridScale = 1024.0;  // largest |W|: lo parts stay normal f16 numbers
constexpr size_t kGridRecBytes = (size_t)512 << 20;  // ray records of one launch
constexpr size_t kGridPartialBytes = (size_t)1 << 30;  // of the splits' partials
// FP32 additions into one partial: of random phasors N lose 1.8e-8 sqrt(N) of the sum
// (4e-7 here, below what one-block segments lose in the tensor cores; 3.3e-6 at 32768).
constexpr int kGridMaxAdds = 512;
constexpr size_t kGridMaxTiles = 4096;               // at least 2048 rays per launch fit then

// ---- order of the screen points -------------------------------------------------

__device__ __forceinline__ const double* coord(const PixDev& p, int c) {
    return c == 0 ? p.x : (c == 1 ? p.y : p.z);
}

// As summary_kernel, up to N screens per launch (nine screens of a batch: 122 us one
// after another, 15 in one launch; a single one is bound by its latency).
template <int N>
struct ProbeBatch {
    ProbeArgs s[N];
};

template <int N>
__global__ void __launch_bounds__(256)
    grid_probe_kernel(const __grid_constant__ ProbeBatch<N> batch) {
    const ProbeArgs& A = solve_of_block(batch.s);
    const PixDev& p = A.pix;
    const int m = A.m, block = (int)blockIdx.x - A.first;
    GridProbe* const out = A.probe;
    const double lend = *A.first_change;
    if (!(lend >= 2.0 && lend <= 0.5 * m)) return;  // len stays 0
    const int len = (int)lend;
    if (m % len != 0) return;
    const int inner = p.x[1] != p.x[0] ? 0 : (p.y[1] != p.y[0] ? 1 : 2);
    if (block == 0 && threadIdx.x == 0) {
        out->len = len;
        out->inner = inner;
    }
    const int t0 = block * 256 + threadIdx.x, step = A.blocks * 256;
    int bad = 0, mask = 0;
    for (int q = t0; q < m; q += step) {
        const int i = q / len, l = q - i * len;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double* a = coord(p, c);
            const double w = a[q];
            bad |= w != a[c == inner ? l : i * len];
            if (c != inner) mask |= (w != a[0]) << c;
        }
    }
    bad = __any_sync(0xffffffffu, bad);
    mask = __reduce_or_sync(0xffffffffu, (unsigned)mask);
    const int lane = threadIdx.x & 31;
    if (lane == 0) {
        if (bad) atomicOr(&out->bad, 1);
        if (mask) atomicOr(&out->outer_mask, mask);
    }
    // Half extents of every tile of every size, one warp per tile. Sizes and axes
    // share the warps' turns, so that a small screen takes one of them.
    const int warp = t0 >> 5, warps = step >> 5;
    int base = 0;  // tiles of the sizes and axes before
    for (int axis = 0; axis < 2; ++axis)
        for (int k = 0; k < kGridSizes; ++k) {
            const int count = axis ? len : m / len, size = kGridSpan << k;
            const int tiles = (count + size - 1) / size;
            for (int t = (warp + warps - base % warps) % warps; t < tiles; t += warps) {
                double half = 0.0;
                for (int c = 0; c < 3; ++c) {
                    if ((c == inner) != (axis == 1)) continue;
                    const double* a = coord(p, c);
                    double lo = INFINITY, hi = -INFINITY;
                    for (int q = t * size + lane; q < min(count, (t + 1) * size); q += 32) {
                        const double w = a[axis ? q : q * len];
                        lo = fmin(lo, w);
                        hi = fmax(hi, w);
                    }
                    for (int o = 16; o > 0; o >>= 1) {
                        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
                    }
                    half = fmax(half, 0.5 * (hi - lo));
                }
                if (lane == 0)
                    atomicMax(&out->extent[axis][k], (unsigned long long)__double_as_longlong(half));
            }
            base += tiles;
        }
    static_assert(sizeof(GridProbe) % 8 == 0, "copied by 8-byte words");
    if (last_block(A.ticket, A.blocks) && threadIdx.x < sizeof(GridProbe) / 8)
        reinterpret_cast<unsigned long long*>(A.host_probe)[threadIdx.x] =
            __ldcg(reinterpret_cast<const unsigned long long*>(out) + threadIdx.x);
}

// One block per tile: the axis coordinates of its points and their mid-range.
__global__ void __launch_bounds__(kTileM) grid_axes_kernel(const double* __restrict__ src_m,
                                                           size_t stride_m, int nm, int m_tiles,
                                                           int span_m,
                                                           const double* __restrict__ src_n,
                                                           size_t stride_n, int nn, int span_n,
                                                           double* __restrict__ axes) {
    const bool is_m = (int)blockIdx.x < m_tiles;
    const int t = is_m ? blockIdx.x : blockIdx.x - m_tiles;
    const int size = is_m ? span_m : span_n, count = is_m ? nm : nn;
    const int q = t * size + threadIdx.x;
    double lo = INFINITY, hi = -INFINITY;
    if ((int)threadIdx.x < size && q < count) {
        const double w = is_m ? src_m[q * stride_m] : src_n[q * stride_n];
        axes[is_m ? q : nm + q] = w;
        lo = hi = w;
    }
    __shared__ double s[8][2];
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        s[threadIdx.x >> 5][0] = lo;
        s[threadIdx.x >> 5][1] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) {
            lo = fmin(lo, s[w][0]);
            hi = fmax(hi, s[w][1]);
        }
        axes[nm + nn + blockIdx.x] = 0.5 * (lo + hi);
    }
}

// ---- ray records ------------------------------------------------------------------

// Per ray and tile (64 bytes; a / b: row / column axis; lengths times
// GridPlan::unit):
//   {La hi, Lb hi, La lo, Lb lo}   L = 2 h A turns
//   {2A, 2B, h - h0, -q}           q = turns of the second-order term per dS^2
//   {R, W re, W im, -m}            R = frac(k D), W = amplitude at p0, scaled
//   {sa, sb, W2 re, W2 im}         amplitude slopes; second column
struct RecordArgs {
    const double *ra, *rb, *rc, *na, *nb, *nc, *nl;
    const double *w_re, *w_im, *w2_re, *w2_im;
    const double* refs;  // tile references: m_tiles, then n_tiles
    int m_tiles, n_tiles;
    size_t n, pad;       // rays of this launch, rounded up to whole blocks
    double c0;
    double unit;         // GridPlan::unit; what follows is in such lengths
    double h0, kt, kt_lo;
    double scale[2];     // of either amplitude column
};

__global__ void __launch_bounds__(256) grid_records_kernel(RecordArgs g, float4* __restrict__ out) {
    const size_t j = blockIdx.x * (size_t)256 + threadIdx.x;
    if (j >= g.pad) return;
    const int tile = blockIdx.y, mt = tile / g.n_tiles, nt = tile - mt * g.n_tiles;
    float4* o = out + ((size_t)tile * g.pad + j) * 4;
    if (j >= g.n) {
        for (int i = 0; i < 4; ++i) o[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    double al, bl, cl;
    double a = dd_diff(g.refs[mt], g.ra[j], &al), b = dd_diff(g.refs[g.m_tiles + nt], g.rb[j], &bl),
           c = dd_diff(g.c0, g.rc[j], &cl);
    a *= g.unit;  // a power of two: exact
    b *= g.unit;
    c *= g.unit;
    al *= g.unit;
    bl *= g.unit;
    cl *= g.unit;
    double d, unused;
    const double turns = dd_turns<true>(g.kt, g.kt_lo, a, b, c, &d, &unused,
                                        2.0 * (a * al + b * bl + c * cl));
    const double inv = 1.0 / d, h = 0.5 * g.kt * inv;
    const double na = g.na[j], nb = g.nb[j], nc = g.nc[j];
    const double nu = (na * a + nb * b + nc * c) * inv;
    const double obl = g.nl[j] + nu;
    const double w = obl * inv, w1 = w * g.scale[0];
    const double la = 2.0 * h * a, lb = 2.0 * h * b;
    const float lah = (float)la, lbh = (float)lb;
    o[0] = make_float4(lah, lbh, (float)(la - (double)lah), (float)(lb - (double)lbh));
    o[1] = make_float4((float)(2.0 * a), (float)(2.0 * b), (float)(h - g.h0),
                       (float)(-0.25 * h * inv * inv));
    o[2] = make_float4((float)(turns - rint(turns)), (float)(g.w_re[j] * w1),
                       (float)(g.w_im[j] * w1), (float)(-0.5 * (1.0 + nu / obl) * inv * inv));
    float4 e = make_float4((float)(na * inv / obl), (float)(nb * inv / obl), 0.f, 0.f);
    if (g.w2_re) {
        const double w2 = w * g.scale[1];
        e.z = (float)(g.w2_re[j] * w2);
        e.w = (float)(g.w2_im[j] * w2);
    }
    o[3] = e;
}

// ---- the product --------------------------------------------------------------------

struct ProductArgs {
    const float4* recs;
    size_t pad;
    int ray_blocks, splits, seg;
    int m_tiles, n_tiles;
    int span_m, span_n;  // rows and columns of a tile in use
    const double *cm, *cn, *refs;
    size_t nm, nn;
    double unit, h0;  // GridPlan::unit; turns per squared such length
    float* partial;  // [splits][m_pad][n_pad], in the order of partial_at
    int m_pad, n_pad;
    int* err;
    uint32_t wait_limit, stall;
};

// Offset from the tile's reference (in GridPlan::unit) of row `row` of row tile t,
// of column `col` of column tile t; 0 outside the rows and columns in use.
__device__ __forceinline__ double row_offset(const ProductArgs& g, int t, int row) {
    const size_t i = (size_t)t * g.span_m + row;
    return row < g.span_m && i < g.nm ? (g.cm[i] - g.refs[t]) * g.unit : 0.0;
}
__device__ __forceinline__ double col_offset(const ProductArgs& g, int t, int col) {
    const size_t i = (size_t)t * g.span_n + col;
    return col < g.span_n && i < g.nn ? (g.cn[i] - g.refs[g.m_tiles + t]) * g.unit
                                         : 0.0;
}

__device__ __forceinline__ uint32_t neg2(uint32_t v) { return v ^ 0x80008000u; }

__device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {
    const __half2 r = __hmul2(*reinterpret_cast<const __half2*>(&a),
                              *reinterpret_cast<const __half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&r);
}

// A pair-row: a row of A (.x) and a row of B (.y), or two rows of A (ZZ),
// evaluated together in packed instructions.
struct PairRow {
    float2 kh, khn, kl, pp, sq;
    __device__ __forceinline__ void set(double ux, double uy, double h0) {
        float hx, lx, hy, ly, fx, fy;
        split_coord(ux, h0, &hx, &lx, &fx);
        split_coord(uy, h0, &hy, &ly, &fy);
        kh = make_float2(hx, hy);
        khn = make_float2(-hx, -hy);
        kl = make_float2(lx, ly);
        pp = make_float2(fx, fy);
        sq = make_float2((float)(ux * ux), (float)(uy * uy));
    }
    // Phasors (c, s) of one ray record and the first-order factors ex, ey. The
    // B row's phasor is W; ZZ: a second A phasor. AMP: the amplitude varies
    // along the tile.
    template <bool ZZ, bool AMP>
    __device__ __forceinline__ void ray(float4 v0, float4 v1, float4 v2, float4 v3, bool col,
                                        float& cx, float& sx, float& cy, float& sy, float& ex,
                                        float& ey) const {
        const float2 rh = ZZ ? f2(v0.x) : make_float2(v0.x, v0.y);
        const float2 rl = ZZ ? f2(v0.z) : make_float2(v0.z, v0.w);
        const float2 ab = ZZ ? f2(v1.x) : make_float2(v1.x, v1.y);
        const float2 ds = __ffma2_rn(kh, ab, sq);    // dS, dT
        const float2 qd = __fmul2_rn(f2(v1.w), ds);  // -q dS, -q dT
        const float2 small = __ffma2_rn(qd, ds, __fmul2_rn(f2(v1.z), sq));
        float2 p0 = __fadd2_rn(pp, small);
        if (!ZZ) p0 = __fadd2_rn(p0, make_float2(0.f, v2.x));
        const float2 t = pair_turns2(kh, khn, kl, p0, rh, rl);
        const float2 th = __fmul2_rn(t, f2(6.28318530717958647692f));
        __sincosf(th.x, &sx, &cx);
        __sincosf(th.y, &sy, &cy);
        ex = ds.x;
        ey = ZZ ? ds.y : qd.y * 12.566370614359172f;
        float2 f = f2(1.f);
        if (AMP) {
            const float2 sl = ZZ ? f2(v3.x) : make_float2(v3.x, v3.y);
            f = __ffma2_rn(kh, sl, __ffma2_rn(f2(v2.w), ds, f2(1.f)));
            cx *= f.x;
            sx *= f.x;
        }
        if (ZZ) {
            if (AMP) {
                cy *= f.y;
                sy *= f.y;
            }
        } else {
            const float wr0 = col ? v3.z : v2.y, wi0 = col ? v3.w : v2.z;
            const float ar = AMP ? wr0 * f.y : wr0, ai = AMP ? wi0 * f.y : wi0;
            const float co = cy, si = sy;
            cy = cmul_re(ar, ai, co, si);  // W
            sy = cmul_im(ar, ai, co, si);
        }
    }
};

// (c, s) of two rays -> f16 hi, lo and hi times the factors (e0, e1); returns these.
__device__ __forceinline__ uint32_t split_pair(const float (&c)[2], const float (&s)[2], float e0,
                                               float e1, uint32_t* h, uint32_t* l, uint32_t* e,
                                               int re, int im) {
    split16x2(c[0], c[1], &h[re], &l[re]);
    split16x2(s[0], s[1], &h[im], &l[im]);
    const uint32_t f = pack16x2(e0, e1);
    e[re] = mul2(h[re], f);
    e[im] = mul2(h[im], f);
    return f;
}

// Producer warps of a CTA of the pair, narrow form. A warp fills 16-byte chunks
// (four rays) of pair-rows: warp w < 8 chunk w of the pair-rows 0..63 (A rows with
// the CTA's 64 columns), warps 8..11 (ZZ) two chunks each of the pair-rows
// (64 + r, 96 + r) of A alone. Inside a chunk the contraction runs (re j, re j+1,
// im j, im j+1) over ray pairs, in both operands, so that the real-part and
// imaginary-part rows of B hold the same words in another order (and one sign).
// Rows and columns past the screen's edge hold the phasors of the tile's
// reference point: they only reach accumulators nobody reads.
template <bool ZZ, bool AMP>
__device__ __forceinline__ void grid_producer(const ProductArgs& g, int c0, int r, int mt, int nt,
                                              int col, uint32_t half, int nrb,
                                              unsigned char* tiles, uint32_t full_lead,
                                              uint64_t* empty, uint64_t* ray_full,
                                              uint64_t* ray_empty, unsigned char* rays_smem,
                                              volatile int* flag) {
    using namespace sm100;
    using F = Form<kFormNarrow>;
    constexpr int NE = ZZ ? 1 : 2;   // pair-rows per thread
    constexpr int NCH = ZZ ? 2 : 1;  // chunks per thread
    PairRow row[NE];
    const int cta_row = (mt & 1) * 128;
#pragma unroll
    for (int e = 0; e < NE; ++e) {
        const double ux = row_offset(g, mt >> 1, cta_row + (ZZ ? 64 + r : r + 32 * e));
        const double uy = ZZ ? row_offset(g, mt >> 1, cta_row + 96 + r)
                             : col_offset(g, nt, 64 * half + r + 32 * e);
        row[e].set(ux, uy, g.h0);
    }
    for (int i = 0; i < nrb; ++i) {
        const int s = i % F::kStages, rb = i % F::kRayBufs;
        bool ok = mbar_wait(&ray_full[rb], (uint32_t)(i / F::kRayBufs) & 1u, g.wait_limit);
        ok = ok && mbar_wait(&empty[s], ((uint32_t)(i / F::kStages) & 1u) ^ 1u, g.wait_limit);
        if (!__all_sync(0xffffffffu, ok)) {
            *flag = 1;
            return;
        }
        unsigned char* base = tiles + (size_t)s * F::kStage;
        const float4* sr = reinterpret_cast<const float4*>(rays_smem + rb * F::kRayBytes);
#pragma unroll
        for (int ch = 0; ch < NCH; ++ch) {
            const int c = c0 + ch;
            // A rows of .x and (ZZ) of .y; B points of .y: four words per tile.
            uint32_t ah[2][4], al[2][4], ae[2][4], bh[2][4], bl[2][4], be[2][4];
#pragma unroll
            for (int pr = 0; pr < 2; ++pr) {
                float cx[2][2], sx[2][2], cy[2][2], sy[2][2], ex[2][2], ey[2][2];  // [e][ray]
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float4* rec = sr + 4 * (4 * c + 2 * pr + u);
                    const float4 v0 = rec[0], v1 = rec[1], v2 = rec[2];
                    float4 v3 = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (AMP || (!ZZ && col)) v3 = rec[3];
#pragma unroll
                    for (int e = 0; e < NE; ++e)
                        row[e].template ray<ZZ, AMP>(v0, v1, v2, v3, col, cx[e][u], sx[e][u],
                                                     cy[e][u], sy[e][u], ex[e][u], ey[e][u]);
                }
#pragma unroll
                for (int e = 0; e < NE; ++e) {
                    const int k = 2 * pr;
                    split_pair(cx[e], sx[e], ex[e][0], ex[e][1], ah[e], al[e], ae[e], k, k + 1);
                    split_pair(cy[e], sy[e], ey[e][0], ey[e][1], ZZ ? ah[1] : bh[e],
                               ZZ ? al[1] : bl[e], ZZ ? ae[1] : be[e], k, k + 1);
                }
            }
            auto put = [&](int tile, uint32_t row, uint32_t a, uint32_t b, uint32_t d, uint32_t e) {
                *reinterpret_cast<uint4*>(base + tile * kGA + sw128(row, c)) =
                    make_uint4(a, b, d, e);
            };
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const uint32_t row = (uint32_t)((ZZ ? 64 : 0) + r + 32 * k);
                put(0, row, ah[k][0], ah[k][1], ah[k][2], ah[k][3]);
                put(1, row, al[k][0], al[k][1], al[k][2], al[k][3]);
                put(2, row, ae[k][0], ae[k][1], ae[k][2], ae[k][3]);
            }
            if (!ZZ) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    // Point j: (Re W, -Im W) in row j, (Im W, Re W) in row 64 + j;
                    // and the same of i E W, whose real part is -E Im W (be
                    // holds E Re W, E Im W).
                    const uint32_t row = (uint32_t)(r + 32 * k);
                    const uint32_t(&h)[4] = bh[k], (&l)[4] = bl[k], (&o)[4] = be[k];
                    put(3, row, h[0], neg2(h[1]), h[2], neg2(h[3]));
                    put(3, 64 + row, h[1], h[0], h[3], h[2]);
                    put(4, row, l[0], neg2(l[1]), l[2], neg2(l[3]));
                    put(4, 64 + row, l[1], l[0], l[3], l[2]);
                    const uint32_t n1 = neg2(o[1]), n3 = neg2(o[3]);
                    put(5, row, n1, neg2(o[0]), n3, neg2(o[2]));
                    put(5, 64 + row, o[0], n1, o[2], n3);
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

// Producer warps of the wide form: warp w takes rays 8 (w % 4) .. + 7 of the
// stage for the pair-rows 64 (w / 4) .. + 63 (A row and column of the same
// number). Lanes r and r + 8 hold the same pair-row and four rays each, so that
// 16 lanes' 8-byte stores cover eight rows' 16-byte words: no bank conflicts, and
// a record is read once for eight rays x 16 lanes.
template <bool AMP>
__device__ __forceinline__ void grid_producer_wide(const ProductArgs& g, int w, int lane, int mt,
                                                   int nt, int col, uint32_t half, int nrb,
                                                   unsigned char* tiles, uint32_t full_lead,
                                                   uint64_t* empty, uint64_t* ray_full,
                                                   uint64_t* ray_empty, unsigned char* rays_smem,
                                                   volatile int* flag) {
    using namespace sm100;
    using F = Form<kFormWide>;
    constexpr int NE = 2;  // pair-rows at a time (1: 6.68, 2: 6.50, 4: 7.85 ms)
    const int sub = (lane >> 3) & 1, oct = w & 3;
    const int row0 = 64 * (w >> 2) + (lane & 7) + ((lane & 16) >> 1);  // + 16 e
    PairRow row[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
        row[e].set(row_offset(g, mt >> 1, (mt & 1) * 128 + row0 + 16 * e),
                   col_offset(g, nt, 128 * half + row0 + 16 * e), g.h0);
    // This thread's 8 bytes of the real and the imaginary 16-byte word of row 0.
    const uint32_t at_re = sw128(row0, oct) + 8 * sub, at_im = sw128(row0, 4 + oct) + 8 * sub;
    for (int i = 0; i < nrb; ++i) {
        const int s = i % F::kStages, rb = i % F::kRayBufs;
        bool ok = mbar_wait(&ray_full[rb], (uint32_t)(i / F::kRayBufs) & 1u, g.wait_limit);
        ok = ok && mbar_wait(&empty[s], ((uint32_t)(i / F::kStages) & 1u) ^ 1u, g.wait_limit);
        if (!__all_sync(0xffffffffu, ok)) {
            *flag = 1;
            return;
        }
        unsigned char* base = tiles + (size_t)s * F::kStage;
        const float4* sr = reinterpret_cast<const float4*>(rays_smem + rb * F::kRayBytes) +
                           4 * (8 * oct + 4 * sub);
#pragma unroll
        for (int e0 = 0; e0 < 4; e0 += NE) {
            uint32_t ah[NE][4], al[NE][4], ae[NE][4];  // re, re, im, im
            uint32_t bh[NE][4], bl[NE][4], be[NE][4];
#pragma unroll
            for (int pr = 0; pr < 2; ++pr) {
                float cx[NE][2], sx[NE][2], cy[NE][2], sy[NE][2], ex[NE][2], ey[NE][2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float4* rec = sr + 4 * (2 * pr + u);
                    const float4 v0 = rec[0], v1 = rec[1], v2 = rec[2];
                    float4 v3 = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (AMP || col) v3 = rec[3];
#pragma unroll
                    for (int e = 0; e < NE; ++e)
                        row[e0 + e].template ray<false, AMP>(v0, v1, v2, v3, col, cx[e][u],
                                                             sx[e][u], cy[e][u], sy[e][u],
                                                             ex[e][u], ey[e][u]);
                }
#pragma unroll
                for (int e = 0; e < NE; ++e) {
                    split_pair(cx[e], sx[e], ex[e][0], ex[e][1], ah[e], al[e], ae[e], pr, 2 + pr);
                    split_pair(cy[e], sy[e], ey[e][0], ey[e][1], bh[e], bl[e], be[e], pr, 2 + pr);
                }
            }
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                auto put = [&](int tile, const uint32_t(&v)[4]) {
                    unsigned char* o = base + tile * kGA + 16 * 128 * (e0 + e);
                    *reinterpret_cast<uint2*>(o + at_re) = make_uint2(v[0], v[1]);
                    *reinterpret_cast<uint2*>(o + at_im) = make_uint2(v[2], v[3]);
                };
                put(0, ah[e]);
                put(1, al[e]);
                put(2, ae[e]);
                put(3, bh[e]);
                put(4, bl[e]);
                put(5, be[e]);
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

// Producer warps of the second-order form, as grid_producer_wide's: warp w takes rays
// 8 (w % 2) .. + 7 of the stage for the pair-rows 32 (w / 2) .. + 31.
template <bool AMP>
__device__ __forceinline__ void grid_producer_second(const ProductArgs& g, int w, int lane, int mt,
                                                     int nt, int col, uint32_t half, int nrb,
                                                     unsigned char* tiles, uint32_t full_lead,
                                                     uint64_t* empty, uint64_t* ray_full,
                                                     uint64_t* ray_empty,
                                                     unsigned char* rays_smem,
                                                     volatile int* flag) {
    using namespace sm100;
    using F = Form<kFormSecond>;
    constexpr int NE = 2;
    const int sub = (lane >> 3) & 1, oct = w & 1;
    const int row0 = 32 * (w >> 1) + (lane & 7) + ((lane & 16) >> 1);  // + 16 e
    PairRow row[NE];
#pragma unroll
    for (int e = 0; e < NE; ++e)
        row[e].set(row_offset(g, mt >> 1, (mt & 1) * 128 + row0 + 16 * e),
                   col_offset(g, nt, 128 * half + row0 + 16 * e), g.h0);
    // This thread's 8 bytes of row 0's real and imaginary 16-byte words, in the first
    // (hi, first order) and the second (lo, second order) half of the row.
    uint32_t at[2][2];
#pragma unroll
    for (int k = 0; k < 4; ++k) at[k >> 1][k & 1] = sw128(row0, 2 * k + oct) + 8 * sub;
    for (int i = 0; i < nrb; ++i) {
        const int s = i % F::kStages, rb = i % F::kRayBufs;
        bool ok = mbar_wait(&ray_full[rb], (uint32_t)(i / F::kRayBufs) & 1u, g.wait_limit);
        ok = ok && mbar_wait(&empty[s], ((uint32_t)(i / F::kStages) & 1u) ^ 1u, g.wait_limit);
        if (!__all_sync(0xffffffffu, ok)) {
            *flag = 1;
            return;
        }
        unsigned char* base = tiles + (size_t)s * F::kStage;
        const float4* sr = reinterpret_cast<const float4*>(rays_smem + rb * F::kRayBytes) +
                           4 * (8 * oct + 4 * sub);
        // Words re, re, im, im of hi, lo, first and second order.
        uint32_t a[4][NE][4], b[4][NE][4];
#pragma unroll
        for (int pr = 0; pr < 2; ++pr) {
            float cx[NE][2], sx[NE][2], cy[NE][2], sy[NE][2], ex[NE][2], ey[NE][2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float4* rec = sr + 4 * (2 * pr + u);
                const float4 v0 = rec[0], v1 = rec[1], v2 = rec[2];
                float4 v3 = make_float4(0.f, 0.f, 0.f, 0.f);
                if (AMP || col) v3 = rec[3];
#pragma unroll
                for (int e = 0; e < NE; ++e)
                    row[e].template ray<false, AMP>(v0, v1, v2, v3, col, cx[e][u], sx[e][u],
                                                    cy[e][u], sy[e][u], ex[e][u], ey[e][u]);
            }
            constexpr uint32_t kMinusHalf2 = 0xb800b800u;
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                const uint32_t fx = split_pair(cx[e], sx[e], ex[e][0], ex[e][1], a[0][e], a[1][e],
                                               a[2][e], pr, 2 + pr);
                const uint32_t fy = mul2(split_pair(cy[e], sy[e], ey[e][0], ey[e][1], b[0][e],
                                                    b[1][e], b[2][e], pr, 2 + pr),
                                         kMinusHalf2);
#pragma unroll
                for (int k = pr; k < 4; k += 2) {
                    a[3][e][k] = mul2(a[2][e][k], fx);
                    b[3][e][k] = mul2(b[2][e][k], fy);
                }
            }
        }
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                const uint32_t(&v)[4] = t < 2 ? a[2 * t][e] : b[2 * (t - 2)][e];
                const uint32_t(&w2)[4] = t < 2 ? a[2 * t + 1][e] : b[2 * (t - 2) + 1][e];
                unsigned char* o = base + t * kGA + 16 * 128 * e;
                *reinterpret_cast<uint2*>(o + at[0][0]) = make_uint2(v[0], v[1]);
                *reinterpret_cast<uint2*>(o + at[0][1]) = make_uint2(v[2], v[3]);
                *reinterpret_cast<uint2*>(o + at[1][0]) = make_uint2(w2[0], w2[1]);
                *reinterpret_cast<uint2*>(o + at[1][1]) = make_uint2(w2[2], w2[3]);
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

// Epilogue role (warps 1..4): adds each finished accumulator segment to this
// CTA's 128 rows of the split's partial. The partial is stored in contiguous
// blocks of 32 rows x 16 columns (partial_at), so that 16 columns of a warp's 32
// rows go from TMEM through 2 KB of staging to ONE bulk operation, a store for
// the split's first segment and an FP32 add at the memory side (round to nearest)
// for the others. (A 128-byte operation per row kept the bulk unit busy longer
// than a short segment's products: 2^20 rays x 512^2 points took 32.8 ms with
// segments of one block and 7.8 ms with ten, now 16.8 and 7.5 ms, narrow form.)
// Each block's operations complete before its next segment's start, so the
// partial is s0 + s1 + ... in segment order.
template <int FORM>
__device__ __forceinline__ void grid_drain(const ProductArgs& g, int warp, int lane, int mt,
                                           int sp, int nrb, int seg_len, uint32_t tmem,
                                           uint64_t* acc_full,
                                           uint32_t acc_empty_lead, unsigned char* stage,
                                           volatile int* flag) {
    using namespace sm100;
    using F = Form<FORM>;
    constexpr bool WIDE = F::kWide;
    constexpr int kBlocks = kFN / 16, kBlock = 512;  // blocks per accumulator, floats
    const int qd = warp & 3;
    float* row = g.partial + (((size_t)sp * (g.m_pad / 32) + (size_t)mt * 4 + qd) * (g.n_pad / 16) +
                              (size_t)blockIdx.y * F::kAcc * kBlocks) * kBlock;
    // Segments of the accumulators, as the MMA issuer counts them.
    int drains = (nrb + seg_len - 1) / seg_len;
    if (WIDE) drains += 1 + (max(0, nrb - max(1, seg_len / 2)) + seg_len - 1) / seg_len;
    if (nrb == 0) {
        for (int c = lane; c < F::kAcc * kBlocks * kBlock; c += 32) row[c] = 0.f;
        return;
    }
    int buf = 0;
    for (int q = 0; q < drains; ++q) {
        // Accumulator b's next segment; wide: the second one's ends first.
        const int b = (q & 1) ^ (WIDE ? 1 : 0), seg = q / F::kAcc;
        const bool ok = mbar_wait(&acc_full[b], (uint32_t)(q >> 1) & 1u, g.wait_limit);
        if (!__all_sync(0xffffffffu, ok)) {
            *flag = 1;
            break;
        }
        tc_fence_after();
        float* dst = row + (WIDE ? b * kBlocks * kBlock : 0);
#pragma unroll 1
        for (int c = 0; c < kBlocks; c += 2) {
            float v[32];
            tmem_ld_32cols(tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)(b * kFN + c * 16), v);
            if (c == kBlocks - 2) {  // the accumulator is free again
                tc_fence_before();
                mbar_arrive_cluster(acc_empty_lead + 8u * (uint32_t)b);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (lane == 0) bulk_wait_read_but<kGEpiBufs - 1>();  // the buffer is free again
                __syncwarp();
                unsigned char* sb = stage + buf * kDrainBytes;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float* w = v + 16 * h + 4 * k;
                    reinterpret_cast<float4*>(sb + lane * 64)[k ^ ((lane >> 1) & 3)] =
                        make_float4(w[0], w[1], w[2], w[3]);
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    // The previous segment's operation on this block is performed.
                    bulk_wait_but<F::kAcc * kBlocks - 1>();
                    float* to = dst + (c + h) * kBlock;
                    if (seg == 0)
                        bulk_s2g(to, smem_u32(sb), kDrainBytes);
                    else
                        bulk_add_s2g_f32(to, smem_u32(sb), kDrainBytes);
                    bulk_commit();
                }
                buf = buf + 1 == kGEpiBufs ? 0 : buf + 1;
            }
        }
    }
    bulk_wait_all();
}

// Element (row, column) of a split's partial: blocks of 32 x 16, the 16-byte
// words of a block's row permuted by the row (conflict-free staging writes).
__device__ __forceinline__ size_t partial_at(size_t im, size_t x, int n_pad) {
    const size_t r = im & 31, k = (x & 15) ^ (((r >> 1) & 3) << 2);
    return ((im >> 5) * (size_t)(n_pad >> 4) + (x >> 4)) * 512 + r * 16 + k;
}

template <bool AMP, int FORM>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Form<FORM>::kThreads, 1)
    grid_product_kernel(ProductArgs g) {
    using namespace sm100;
    using F = Form<FORM>;
    constexpr bool WIDE = F::kWide;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char* rays_smem = tiles + kGTiles;
    unsigned char* epi_smem = rays_smem + kGRays;
    uint64_t* full = reinterpret_cast<uint64_t*>(epi_smem + 4 * kGEpiBufs * kDrainBytes);
    uint64_t* empty = full + F::kStages;
    uint64_t* acc_full = empty + F::kStages;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* ray_full = acc_empty + 2;
    uint64_t* ray_empty = ray_full + F::kRayBufs;
    uint64_t* mma_done = ray_empty + F::kRayBufs;  // every issued MMA has completed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
    volatile int* flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int mt = blockIdx.x, sp = blockIdx.z;
    const int col = blockIdx.y / g.n_tiles, nt = blockIdx.y - col * g.n_tiles;
    const uint32_t half = cluster_ctarank(), peer = half ^ 1u;
    const bool leader = half == 0;
    const int rb0 = (int)((long long)g.ray_blocks * sp / g.splits);
    const int rb1 = (int)((long long)g.ray_blocks * (sp + 1) / g.splits);
    // Stages of the split and of a segment.
    constexpr int kPerBlock = kFRays / F::kRays;
    const int nrb = (rb1 - rb0) * kPerBlock, seg = g.seg * kPerBlock;

    if (threadIdx.x == 0) {
        // full and acc_empty are used in the even CTA only: they collect the
        // arrivals of both CTAs' producer and epilogue warps.
        for (int s = 0; s < F::kStages; ++s) {
            mbar_init(&full[s], 2 * F::kProdWarps + (s == 0 ? g.stall : 0u));
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 2 * kFEpiThreads);
        }
        for (int b = 0; b < F::kRayBufs; ++b) {
            mbar_init(&ray_full[b], 1);
            mbar_init(&ray_empty[b], F::kProdWarps);
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
            // Pair MMA issuer: per stage the first-order product and the three
            // of the split phasors, 256x256x16 steps, in two parts of a segment
            // (wide: h = 0 the real, 1 the imaginary part of the field).
            constexpr uint32_t idesc = idesc_f16_f32(256, kFN);
            bool good = true;
            auto wait_acc = [&](int b, int use) {  // use: earlier segments of buffer b
                if (use >= 1 &&
                    !mbar_wait_cluster(&acc_empty[b], (uint32_t)(use - 1) & 1u, g.wait_limit)) {
                    *flag = 1;
                    good = false;
                }
                tc_fence_after();
            };
            // Ends of the accumulators' segments; a wide tile's second one ends its
            // own half a segment earlier. A part is issued first in its segment's
            // last stage and last in the next stage, so that the other part's
            // products of both stages run while it is drained.
            int end0 = min(nrb, seg), end1 = min(nrb, max(1, seg / 2)), q0 = 0, q1 = 0;
            bool new0 = true, new1 = true;
            for (int i = 0; i < nrb && good; ++i) {
                const int s = i % F::kStages;
                if (!mbar_wait_cluster(&full[s], (uint32_t)(i / F::kStages) & 1u, g.wait_limit)) {
                    *flag = 1;
                    break;
                }
                tc_fence_after();
                // First order, (second order,) hi hi, hi lo, lo hi.
                const uint32_t t0 = smem_u32(tiles) + (uint32_t)s * F::kStage;
                constexpr int P = F::kSecond ? 5 : 4, K = F::kSecond ? 2 : 4;
                uint32_t as[5], bs[5];
                if (F::kSecond) {
                    const uint32_t a1 = t0 + kGA, b0 = t0 + 2 * kGA, b1 = t0 + 3 * kGA;
                    as[0] = a1, as[1] = a1 + 64, as[2] = t0, as[3] = t0, as[4] = t0 + 64;
                    bs[0] = b1, bs[1] = b1 + 64, bs[2] = b0, bs[3] = b0 + 64, bs[4] = b0;
                } else {
                    as[0] = t0 + 2 * kGA, as[1] = t0, as[2] = t0, as[3] = t0 + kGA;
                    bs[0] = t0 + 5 * kGA, bs[1] = t0 + 3 * kGA, bs[2] = t0 + 4 * kGA;
                    bs[3] = t0 + 3 * kGA;
                }
                const int first = WIDE && ((new0 && i > 0) || i + 1 == end1);
                for (int h = first, t = 0; t < F::kAcc; ++t, h ^= 1) {
                    const bool fresh = h ? new1 : new0;
                    const int q = h ? q1 : q0, b = WIDE ? h : (q & 1);
                    if (fresh) wait_acc(b, WIDE ? q : q >> 1);
                    if (!good) break;
                    const uint32_t d = tmem + (uint32_t)(b * kFN);
#pragma unroll
                    for (int p = 0; p < P; ++p)
#pragma unroll
                        for (int k = 0; k < K; ++k) {
                            // Wide: A's real (k < K / 2) or imaginary parts meet B's
                            // of the same kind, subtracted for the imaginary
                            // ones, or (h) of the other kind; of i E W (p == 0),
                            // stored as E W, the other way round.
                            const int x = k / (K / 2);
                            const bool swap = WIDE && (h ^ (p == 0));
                            const bool neg =
                                WIDE && (p == 0 ? (h == 0 || x == 1) : (h == 0 && x == 1));
                            umma_f16_pair(d, desc_kmajor_sw128(as[p] + 32u * k),
                                          desc_kmajor_sw128(bs[p] + 32u * (swap ? k ^ (K / 2) : k)),
                                          neg ? idesc | kNegateB : idesc,
                                          (uint32_t)(!fresh | p | k));
                        }
                    const bool last = i + 1 == (h ? end1 : end0);
                    if (last) {
                        umma_commit_pair(smem_u32(&acc_full[b]));
                        umma_commit_pair(mapa_shared(&acc_full[b], peer));
                    }
                    (h ? new1 : new0) = last;
                    (h ? q1 : q0) += last;
                    (h ? end1 : end0) = last ? min(nrb, i + 1 + seg) : (h ? end1 : end0);
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
    } else if (warp <= 4) {
        grid_drain<FORM>(g, warp, lane, mt, sp, nrb, seg, tmem, acc_full, mapa_shared(acc_empty, 0),
                         epi_smem + (warp - 1) * kGEpiBufs * kDrainBytes, flag);
    } else if (warp < 5 + F::kProdWarps) {
        const int w = warp - 5;
        const uint32_t full_lead = mapa_shared(full, 0);
        if constexpr (F::kSecond)
            grid_producer_second<AMP>(g, w, lane, mt, nt, col, half, nrb, tiles, full_lead, empty,
                                      ray_full, ray_empty, rays_smem, flag);
        else if constexpr (WIDE)
            grid_producer_wide<AMP>(g, w, lane, mt, nt, col, half, nrb, tiles, full_lead, empty,
                                    ray_full, ray_empty, rays_smem, flag);
        else if (w < 8)
            grid_producer<false, AMP>(g, w, lane, mt, nt, col, half, nrb, tiles, full_lead, empty,
                                      ray_full, ray_empty, rays_smem, flag);
        else
            grid_producer<true, AMP>(g, 2 * (w - 8), lane, mt, nt, col, half, nrb, tiles, full_lead,
                                     empty, ray_full, ray_empty, rays_smem, flag);
    } else if (lane == 0) {
        // Ray stager: one bulk copy of a stage's records.
        const float4* src =
            g.recs + ((size_t)((mt >> 1) * g.n_tiles + nt) * g.pad + (size_t)rb0 * kFRays) * 4;
        int i = 0;
        for (; i < nrb; ++i) {
            const int rb = i % F::kRayBufs;
            if (i >= F::kRayBufs &&
                !mbar_wait(&ray_empty[rb], (uint32_t)(i / F::kRayBufs - 1) & 1u, g.wait_limit)) {
                *flag = 1;
                break;
            }
            mbar_arrive_expect_tx(&ray_full[rb], F::kRayBytes);
            bulk_g2s(rays_smem + rb * F::kRayBytes, src + (size_t)i * F::kRays * 4, F::kRayBytes,
                     &ray_full[rb]);
        }
        // No copy may still be writing into this CTA's shared memory when it
        // exits: the last ones land whether or not a producer waits for them.
        for (int k = max(0, i - F::kRayBufs); k < i; ++k)
            if (!mbar_wait(&ray_full[k % F::kRayBufs], (uint32_t)(k / F::kRayBufs) & 1u,
                           max(g.wait_limit, kMmaDrainPolls)))
                *flag = 1;
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

// Field of every screen point: the splits' sums in split order, times `scale`
// (i k / (4 pi) over the column's f16 scaling). One column: (Es, Ep) = (pes, pep) A.
// `add`: to what earlier launches' rays left there. Threads run along the columns,
// which are consecutive in the partials.
__global__ void __launch_bounds__(256) grid_reduce_kernel(const float* __restrict__ partial,
                                                          int splits, int m_pad, int n_pad,
                                                          int columns, bool wide, int span_m,
                                                          int span_n, size_t nm, size_t nn,
                                                          bool rows_outer, double2 scale,
                                                          double2 pes, double2 pep, bool add,
                                                          FieldDev out) {
    const size_t idx = blockIdx.x * (size_t)256 + threadIdx.x;
    if (idx >= nm * nn) return;
    const size_t im = idx / nn, in = idx - im * nn;
    // Row and real part's column in the partials; the imaginary part's column is 256
    // (wide) or 64 further.
    const size_t mt = im / span_m, nt = in / span_n, ln = in - nt * span_n;
    const size_t row = mt * kTileM + (im - mt * span_m);
    const size_t at = wide ? nt * 512 + ln : nt * 256 + 128 * (ln >> 6) + (ln & 63);
    const int im_off = (wide ? 256 : 64) / 16 * 512;
    double re[2] = {0.0, 0.0}, ie[2] = {0.0, 0.0};
    for (int c = 0; c < columns; ++c)
        for (int s = 0; s < splits; ++s) {
            const float* e = partial + partial_at((size_t)s * m_pad + row,
                                                  (size_t)c * (n_pad / columns) + at, n_pad);
            re[c] += e[0];
            ie[c] += e[im_off];
        }
    // times i
    for (int c = 0; c < 2; ++c) {
        const double t = re[c], f = c ? scale.y : scale.x;
        re[c] = -ie[c] * f;
        ie[c] = t * f;
    }
    const size_t o = rows_outer ? idx : in * nm + im;
    double f[4] = {re[0], ie[0], re[1], ie[1]};
    if (columns == 1) {
        f[0] = pes.x * re[0] - pes.y * ie[0];
        f[1] = pes.x * ie[0] + pes.y * re[0];
        f[2] = pep.x * re[0] - pep.y * ie[0];
        f[3] = pep.x * ie[0] + pep.y * re[0];
    }
    if (add) {
        f[0] += out.es_re[o];
        f[1] += out.es_im[o];
        f[2] += out.ep_re[o];
        f[3] += out.ep_im[o];
    }
    out.es_re[o] = f[0];
    out.es_im[o] = f[1];
    out.ep_re[o] = f[2];
    out.ep_im[o] = f[3];
}

// ---- host ------------------------------------------------------------------------------

struct Range {
    double lo, hi;
};
Range mul(Range a, Range b) {
    const double v[4] = {a.lo * b.lo, a.lo * b.hi, a.hi * b.lo, a.hi * b.hi};
    return {*std::min_element(v, v + 4), *std::max_element(v, v + 4)};
}

double largest(Range a) { return std::max(std::fabs(a.lo), std::fabs(a.hi)); }

size_t blocks_of(size_t n, size_t size) { return (n + size - 1) / size; }

const double* coord_host(const PixDev& p, int c) { return c == 0 ? p.x : (c == 1 ? p.y : p.z); }

// Bytes of one split's partial.
size_t partial_plane(const GridPlan& g) {
    return (size_t)g.m_tiles * kTileM * g.n_tiles * g.columns *
           (g.form == kFormNarrow ? 1 : 2) * kFN * sizeof(float);
}

double bits_to_double(unsigned long long b) {
    double d;
    std::memcpy(&d, &b, sizeof(d));
    return d;
}

}  // namespace

Status grid_probe_enqueue(std::vector<ProbeArgs>& screens, cudaStream_t stream, int* kernels) {
    for (ProbeArgs& a : screens)
        a.blocks = (int)std::min<size_t>(blocks_of((size_t)a.m, 1024), 296);
    if (screens.size() == 1)
        return launch_solves<1, ProbeBatch<1>>(grid_probe_kernel<1>, screens, stream, kernels);
    return launch_solves<kSolvesPerLaunch, ProbeBatch<kSolvesPerLaunch>>(
        grid_probe_kernel<kSolvesPerLaunch>, screens, stream, kernels);
}

bool grid_plan(const GridProbe& probe, const GridRanges& r, size_t n, size_t m, int columns,
               double tolerance, int num_sms, GridPlan* g) {
    if (probe.len < 2 || probe.bad || !(r.max_amp[0] > 0.0 || r.max_amp[1] > 0.0)) return false;
    const int inner = probe.inner;
    const int mask = probe.outer_mask;
    if (mask != 1 && mask != 2 && mask != 4) return false;
    const int outer = mask == 1 ? 0 : (mask == 2 ? 1 : 2);
    const size_t len = (size_t)probe.len, rows = m / len;

    // Ray-to-point ranges: |p - r| between the boxes, components of p - r.
    Range del[3];
    double d2lo = 0.0, d2hi = 0.0;
    for (int c = 0; c < 3; ++c) {
        del[c] = {r.plo[c] - r.rhi[c], r.phi[c] - r.rlo[c]};
        const double gap = std::max(0.0, std::max(del[c].lo, -del[c].hi));
        d2lo += gap * gap;
        d2hi += largest(del[c]) * largest(del[c]);
    }
    const double dlo = std::sqrt(d2lo), dhi = std::sqrt(d2hi);
    if (!(dlo > 0.0)) return false;
    const double kt = r.k / (2.0 * 3.14159265358979323846);
    // Obliquity factor nl + n.(p - r)/|p - r|.
    Range nd{0.0, 0.0};
    for (int c = 0; c < 3; ++c) {
        const Range u = mul(del[c], {1.0 / dhi, 1.0 / dlo});
        const Range t = mul({r.nlo[c], r.nhi[c]}, {std::max(u.lo, -1.0), std::min(u.hi, 1.0)});
        nd.lo += t.lo;
        nd.hi += t.hi;
    }
    const Range obl{r.nl_lo + nd.lo, r.nl_hi + nd.hi};
    if (!(obl.lo > 0.0 || obl.hi < 0.0)) return false;
    const double omin = std::min(std::fabs(obl.lo), std::fabs(obl.hi)), omax = largest(obl);

    // Form, and rows along the outer or the inner axis: whichever costs less
    // (then whichever leaves the smaller mixed phase).
    bool found = false;
    double best_cost = 0.0, best_e = 0.0;
    // Tiles may use fewer rows (256 >> fm) or columns (of 128 >> fn, or 256; with the
    // second order 256 >> fn - 4) than they have: E falls with either, at the price of
    // the rest, which is still below the general kernel's down to 1/16 of a tile (2^18
    // rays x 256^2 points +-1 mm at 1 m: 10.3 -> 1.07 ms at 10 keV, 12.0 -> 3.6 at 20,
    // 12.3 -> 3.6 at 30).
    const double d2 = dlo * dlo, d3 = d2 * dlo, d5 = d3 * d2;
    constexpr int kSpans = 2 * kGridSizes;
    for (int i = 0; i < 2 * kGridSizes * kSpans; ++i) {
        const bool swap = i & 1;
        const int fm = (i >> 1) % kGridSizes, fn = (i >> 1) / kGridSizes;
        const int form = fn < kGridSizes - 1 ? kFormNarrow
                                             : (fn == kGridSizes - 1 ? kFormWide : kFormSecond);
        const int am = swap ? inner : outer, an = swap ? outer : inner;
        const size_t nm = swap ? len : rows, nn = swap ? rows : len;
        const int tile_n = form == kFormNarrow ? Form<kFormNarrow>::kTileN
                                               : Form<kFormWide>::kTileN;
        const int zm = kGridSizes - 1 - fm;  // sizes of the rows and columns in use
        const int zn = form == kFormNarrow ? kGridSizes - 2 - fn
                                           : (form == kFormWide ? kGridSizes - 1 : kSpans - 1 - fn);
        const int span_m = kGridSpan << zm, span_n = kGridSpan << zn;
        const size_t mt = blocks_of(nm, span_m), nt = blocks_of(nn, span_n);
        if (mt * nt > kGridMaxTiles) continue;
        const double em = bits_to_double(probe.extent[swap ? 1 : 0][zm]);
        const double en = bits_to_double(probe.extent[swap ? 0 : 1][zn]);
        // |dS| = |u| |(p - r) + (p0 - r)| with |p0 - r| <= |p - r|max - |u|max
        // when the tile lies inside the screen's range.
        const double pm = largest(del[am]), pn = largest(del[an]);
        const double ds = em * (2.0 * pm - em), dt = en * (2.0 * pn - en);
        const double e = r.k * ds * dt / (4.0 * d3);
        const double big = std::max(ds, dt);
        // What 1 + iE (- E^2 / 2) leaves out of exp(i phase): E^2 / 2 (E^3 / 6), and the
        // next order of the mixed phase, 3/4 E (dS + dT) / D^2. Both at the far corner of
        // a tile and of the ray box: on a screen beside the rays' axis nearly every ray
        // has that E, and a focus on a tile's corner then has that error (rays of +-0.05
        // mm, 5.9 mm off both axes at 1 m, 1 + iE: 1.5e-4 at E = 0.019). A tenth of the
        // tolerance is about the general kernel's error on coherent fields.
        const double left = form == kFormSecond ? e * e * e / 6.0 : 0.5 * e * e;
        if (!(left + 0.75 * e * (ds + dt) / d2 <= kGridShare * tolerance)) continue;
        // The first-order operands' roundings, 3.5e-4 E of a pair, random over the rays.
        if (!(e <= kGridMostE * tolerance)) continue;
        if (!(big / d2 <= 1e-2)) continue;
        // Linear phase: an exact FP32 product up to 2^21 turns.
        if (!(kt / dlo * std::max(em * pm, en * pn) < 1.9e6)) continue;
        // FP32 terms: u^2 (h - h0) and the dropped third order of the root.
        if (!(0.5 * kt * (1.0 / dlo - 1.0 / dhi) * std::max(em * em, en * en) <= 24.0)) continue;
        if (!(kt * big * big * big / (16.0 * d5) <= 1e-7)) continue;
        // Amplitude: first order along each axis, mixed terms dropped.
        const double sm = largest({r.nlo[am], r.nhi[am]}) * em / (dlo * omin);
        const double sn = largest({r.nlo[an], r.nhi[an]}) * en / (dlo * omin);
        const double mq = 0.5 * (1.0 + largest(nd) / omin) * big / d2;
        if (!(sm <= 0.25 && sn <= 0.25 && sm * sn <= 1e-6 && (sm + sn) * mq <= 1e-6 &&
              mq * mq <= 1e-7))
            continue;
        // Product: 36e12 pairs/s of the padded screen in the narrow form (2^20 rays x
        // 512^2 points, one column). Wide: 0.85 of its time (6.3 to 7.5 ms there,
        // kernels alone) and 18 us more for twice the partials per tile (first to
        // last kernel, narrow and wide: 101 and 115 us at 10^4 rays x 256^2, 135 and
        // 141 at 3 10^4, 253 and 244 at 10^5; 289 and 265 at 3 10^4 x 512^2). With the
        // second order 1.1 of the narrow form's (8.6 ms there at 0.5 m), and the same 18 us.
        const double area = (double)mt * kTileM * (double)nt * tile_n;
        const double rel = form == kFormNarrow ? 1.0 : (form == kFormWide ? 0.85 : kSecondCost);
        const double cost = area * columns * (double)n / 36e12 * rel +
                            (form == kFormNarrow ? 0.0 : 18e-6);
        if (found && !(cost < best_cost || (cost == best_cost && e < best_e))) continue;
        found = true;
        best_cost = cost;
        best_e = e;
        g->m_axis = am;
        g->n_axis = an;
        g->c_axis = 3 - am - an;
        g->rows_outer = swap == 0;
        g->nm = nm;
        g->nn = nn;
        g->form = form;
        g->span_m = span_m;
        g->span_n = span_n;
        g->m_tiles = (int)mt;
        g->n_tiles = (int)nt;
        g->e_bound = e;
        // The first-order factors dS and 4 pi q dT (whose product is E) and their
        // products with phasors of up to 1 and kGridScale are f16 numbers: normal
        // from 6e-5, finite to 65504. In mm dS and the other factor, k dT / (4 D^3),
        // may lie anywhere (1 mm from an aperture the second passes 65504 times
        // over, 50 m from one it is below 6e-5). With the largest dS within 1 .. 4
        // the other operand is at most kGridScale E, and what either loses below 6e-5 is
        // 3e-8 of its own largest value or of kGridScale.
        const int half_exp = ds > 0.0 ? (int)std::floor(0.5 * std::ilogb(ds)) : 0;
        g->unit = std::ldexp(1.0, -std::clamp(half_exp, -100, 100));
        // Below 2^-22 the change of the amplitude along a tile is lost in the
        // split phasors' own rounding.
        g->amp = std::max(sm, sn) + mq > 2.384185791015625e-7;
    }
    if (!found) return false;
    // Measured rates of the general path: 1.6e12 pairs/s (1.2e12 with two columns)
    // after 0.2 ms of sorting tiles and rays that the product does without (0.34 ms
    // in all against 0.10 on 1024 rays x 40 x 51 points).
    const double t_general = 2e-4 + (double)m * (double)n / (columns == 1 ? 1.6e12 : 1.2e12);
    if (best_cost > t_general) return false;
    const double d0 = std::sqrt((r.pc[0] - r.rc[0]) * (r.pc[0] - r.rc[0]) +
                                (r.pc[1] - r.rc[1]) * (r.pc[1] - r.rc[1]) +
                                (r.pc[2] - r.rc[2]) * (r.pc[2] - r.rc[2]));
    const long double kt_ld =
        (long double)r.k / (2.0L * 3.14159265358979323846264338327950288L);
    g->k = r.k;
    g->kt = (double)kt_ld;
    g->kt_lo = (double)(kt_ld - (long double)g->kt);
    g->h0 = g->kt / (2.0 * d0);
    g->c0 = r.plo[g->c_axis];
    g->inner_len = len;
    g->columns = columns;
    g->n = n;
    // Either column by its own largest amplitude: one scale for both left a column
    // 1e-7 times the other's with 3e-4 of error, one 1e-10 times with none of its bits.
    for (int c = 0; c < columns; ++c) {
        g->inv_scale[c] = r.max_amp[c] > 0.0
                              ? kGridScale / (1.4142135623730951 * r.max_amp[c] * omax / dlo)
                              : 1.0;
        if (!std::isfinite(g->inv_scale[c])) return false;
    }
    if (!std::isfinite(g->h0)) return false;
    // Blocks per segment. The tensor cores truncate when they accumulate, 16 MMAs
    // per block: on top of 3.5e-7 (sine and cosine of both factors) the error
    // against 64 bits is 4.7e-7, 6.5e-7, 8.3e-7 and 2.4e-6 of the field at 1, 2,
    // 3 and 10 blocks (14.9, 8.6, 7.7 and 6.3 ms on 2^20 rays x 512^2 points).
    // The persistent kernel's error grows with its FP32 residual phases, whose
    // mean over the whole ray set is about
    //     phase = k (rho^2 + 2 v rho) / (2 d),
    // rho the rays' spread and v the radius of its 256-point tiles: measured
    // 3e-7, 5.3e-7, 1.2e-6, 1.6e-6 and 6e-6 at 5, 7, 14, 18 and from 27 rad on.
    // Below 7 rad the product would be the less exact of the two.
    const double side = 16.0 * std::sqrt((r.phi[g->m_axis] - r.plo[g->m_axis]) *
                                         (r.phi[g->n_axis] - r.plo[g->n_axis]) / (double)m);
    const double phase =
        r.k * (r.spread2 + 0.6 * side * std::sqrt(r.spread2)) / (2.0 * d0);
    if (phase < 7.0) return false;
    // The second order makes it 20 MMAs per block.
    const bool second = g->form == kFormSecond;
    g->seg = phase < 12.0 ? 1 : phase < 24.0 ? (second ? 2 : 3) : (second ? 8 : 10);
    // Rays per launch: what their records' memory allows, and what `cap` splits can sum
    // in kGridMaxAdds segments each (a launch is added to the field in FP64).
    const size_t tiles = (size_t)g->m_tiles * g->n_tiles;
    const size_t cap = std::max<size_t>(1, kGridPartialBytes / partial_plane(*g));
    const size_t segs = (size_t)kGridMaxAdds * g->seg;  // blocks per split
    const size_t fit = std::max<size_t>(kGridRecBytes / (tiles * 64) / kFRays, 64);
    g->ray_blocks = (int)blocks_of(n, kFRays);
    const size_t blocks = std::min<size_t>((size_t)g->ray_blocks, std::min(fit, cap * segs));
    g->chunk_rays = blocks * kFRays;
    // Ray splits: whole waves of CTA pairs, a split at least ten blocks and at most
    // kGridMaxAdds segments long.
    const size_t units = std::max(1, num_sms / 2), work = tiles * columns;
    const size_t least = blocks_of(blocks, segs);
    const size_t most = std::min(cap, std::max(least, blocks / 10));
    size_t s = std::max<size_t>(1, units / work);
    if (work > units || s < least) {
        double best = 1e300;
        for (size_t t = least; t < least + std::max<size_t>(8, units / work); ++t) {
            const double waves = (double)blocks_of(work * t, units) * units / (double)(work * t);
            const double cost =
                waves + 0.01 * (double)(t - least) * std::min(1.0, (double)units / work);
            if (cost < best) {
                best = cost;
                s = t;
            }
        }
    }
    g->splits = (int)std::min(s, most);
    return true;
}

Status grid_axes_enqueue(const GridPlan& g, cudaStream_t stream) {
    const size_t sm = g.rows_outer ? g.inner_len : 1, sn = g.rows_outer ? 1 : g.inner_len;
    grid_axes_kernel<<<g.m_tiles + g.n_tiles, kTileM, 0, stream>>>(
        coord_host(g.pix, g.m_axis), sm, (int)g.nm, g.m_tiles, g.span_m, coord_host(g.pix, g.n_axis), sn,
        (int)g.nn, g.span_n, g.axes);
    XK_CUDA_TRY(cudaGetLastError());
    return Status::Ok();
}

void grid_sizes(const GridPlan& g, size_t* recs, size_t* partial) {
    const size_t tiles = (size_t)g.m_tiles * g.n_tiles;
    *recs = std::max(*recs, tiles * g.chunk_rays * 64);
    *partial = std::max(*partial, g.splits * partial_plane(g));
}

Status grid_reserve(size_t recs, size_t partial, GridWorkspace& ws) {
    XK_TRY(ws.recs.ensure(recs));
    XK_TRY(ws.partial.ensure(partial));
    return Status::Ok();
}

Status grid_enqueue(const GridPlan& g, GridWorkspace& ws, int* err, uint32_t wait_limit,
                    bool stall, cudaStream_t stream, int* kernels) {
    size_t rec_bytes = 0, partial_bytes = 0;
    grid_sizes(g, &rec_bytes, &partial_bytes);
    XK_TRY(grid_reserve(rec_bytes, partial_bytes, ws));
    const double* rays[12];
    std::memcpy(rays, &g.rays, sizeof(rays));
    const double* axes_m = g.axes;
    ProductArgs p{};
    p.recs = ws.recs.as<float4>();
    p.splits = g.splits;
    p.seg = g.seg;
    p.m_tiles = g.m_tiles;
    p.n_tiles = g.n_tiles;
    p.span_m = g.span_m;
    p.span_n = g.span_n;
    p.cm = axes_m;
    p.cn = axes_m + g.nm;
    p.refs = axes_m + g.nm + g.nn;
    p.nm = g.nm;
    p.nn = g.nn;
    p.unit = g.unit;
    p.h0 = g.h0 / (g.unit * g.unit);
    p.partial = ws.partial.as<float>();
    p.m_pad = g.m_tiles * kTileM;
    p.n_pad = g.n_tiles * g.columns * (g.form == kFormNarrow ? 1 : 2) * kFN;
    p.err = err;
    p.wait_limit = wait_limit;
    p.stall = stall ? 1 : 0;
    void (*const kernels_of[3][2])(ProductArgs) = {
        {grid_product_kernel<false, kFormNarrow>, grid_product_kernel<true, kFormNarrow>},
        {grid_product_kernel<false, kFormWide>, grid_product_kernel<true, kFormWide>},
        {grid_product_kernel<false, kFormSecond>, grid_product_kernel<true, kFormSecond>}};
    const auto kern = kernels_of[g.form][g.amp ? 1 : 0];
    static_assert(Form<kFormSecond>::kThreads == Form<kFormWide>::kThreads, "threads");
    const int threads = g.form == kFormNarrow ? Form<kFormNarrow>::kThreads
                                              : Form<kFormWide>::kThreads;
    // Set on every call: the attribute belongs to the current device's context.
    XK_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGSmem));
    const dim3 grid((unsigned)(2 * g.m_tiles), (unsigned)(g.n_tiles * g.columns),
                    (unsigned)g.splits);
    const double amp = g.k / (4.0 * 3.14159265358979323846);
    for (size_t j0 = 0; j0 < g.n; j0 += g.chunk_rays) {
        const size_t cnt = std::min(g.chunk_rays, g.n - j0), pad = blocks_of(cnt, kFRays) * kFRays;
        RecordArgs a{};
        a.ra = rays[g.m_axis] + j0;
        a.rb = rays[g.n_axis] + j0;
        a.rc = rays[g.c_axis] + j0;
        a.na = rays[3 + g.m_axis] + j0;
        a.nb = rays[3 + g.n_axis] + j0;
        a.nc = rays[3 + g.c_axis] + j0;
        a.nl = g.rays.nl + j0;
        a.w_re = g.amps[0][0] + j0;
        a.w_im = g.amps[0][1] + j0;
        if (g.columns == 2) {
            a.w2_re = g.amps[1][0] + j0;
            a.w2_im = g.amps[1][1] + j0;
        }
        a.refs = p.refs;
        a.m_tiles = g.m_tiles;
        a.n_tiles = g.n_tiles;
        a.n = cnt;
        a.pad = pad;
        a.c0 = g.c0;
        a.unit = g.unit;
        a.h0 = p.h0;
        a.kt = g.kt / g.unit;
        a.kt_lo = g.kt_lo / g.unit;
        for (int c = 0; c < 2; ++c) a.scale[c] = g.inv_scale[c] * g.unit;
        grid_records_kernel<<<dim3((unsigned)blocks_of(pad, 256),
                                   (unsigned)(g.m_tiles * g.n_tiles)), 256, 0, stream>>>(
            a, ws.recs.as<float4>());
        XK_CUDA_TRY(cudaGetLastError());
        p.pad = pad;
        p.ray_blocks = (int)(pad / kFRays);
        kern<<<grid, threads, kGSmem, stream>>>(p);
        XK_CUDA_TRY(cudaGetLastError());
        p.stall = 0;
        grid_reduce_kernel<<<(unsigned)blocks_of(g.nm * g.nn, 256), 256, 0, stream>>>(
            p.partial, g.splits, p.m_pad, p.n_pad, g.columns, g.form != kFormNarrow, g.span_m,
            g.span_n, g.nm, g.nn, g.rows_outer, make_double2(amp / g.inv_scale[0], amp / g.inv_scale[1]),
            make_double2(g.pes[0], g.pes[1]), make_double2(g.pep[0], g.pep[1]), j0 > 0, g.out);
        XK_CUDA_TRY(cudaGetLastError());
        *kernels += 3;
    }
    return Status::Ok();
}

}  // namespace xk
