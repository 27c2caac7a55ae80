// Plain FP64 Kirchhoff path: the reference algorithm run directly in FP64.
//
// Per pair it evaluates the expression of src/waves/diffraction.rs:76-110
// (diffraction_at_pixel). The phase k |p - r| is rounded step by step as the
// reference rounds it (explicit intrinsics, no FMA: one ulp of the path is
// 1e-5 rad), so sin and cos are taken of the same number; the smooth factors
// around them use FMAs and one reciprocal of the path. Each thread accumulates
// its pixels with per-component complex Kahan summation in ray order, as the
// reference does.
//
// The kernel is bound by the FP64 pipe and by issue: 71 FP64 and about 60 other
// instructions per pair. With the library's sincos, square root and two
// divisions it took 408 instructions per pair; on 2^16 rays x 128^2 points
// 16.2 ms then, 5.9 ms now (181 Gpair/s; the 71 FP64 instructions alone need
// 4.1 ms), error against a 64-bit evaluation unchanged (6e-16).
//
// Parallel layout: a CTA owns 128*kF64Ppt screen points; the ray list is cut
// into `splits` contiguous ranges (grid.y) when there are too few screen
// points to fill 148 SMs. Each range writes its compensated partial sum; a
// second kernel adds the partials in range order with Kahan summation.
// Rays are staged through shared memory kF64Stage at a time so every ray
// record is read from L2 once per CTA.

#include "xk_internal.cuh"

namespace xk {
namespace {

constexpr int kF64Threads = 128;
constexpr int kF64Ppt = 2;      // screen points per thread
constexpr int kF64Ctas = 4;     // CTAs per SM (108 registers)
constexpr int kF64Stage = 32;   // rays per shared-memory stage
constexpr int kRecDoubles = 16; // 128-byte ray record

// Packed ray record: x y z nx ny nz nl es_re es_im ep_re ep_im k kf pad*3.
struct __align__(16) RayRec64 {
    double x, y, z, nx, ny, nz, nl, es_re, es_im, ep_re, ep_im, k, kf, pad0, pad1, pad2;
};
static_assert(sizeof(RayRec64) == kRecDoubles * 8, "ray record is 128 bytes");

// k = E / CHBAR * 1e7 and k/(4*pi) are pure functions of the ray, so they
// are hoisted out of the pair loop; both are rounded exactly as the
// reference rounds them (diffraction.rs:89,97).
__global__ void f64_pack_kernel(RaysDev r, size_t n, RayRec64* __restrict__ out) {
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    RayRec64 o;
    o.x = r.x[i];
    o.y = r.y[i];
    o.z = r.z[i];
    o.nx = r.nx[i];
    o.ny = r.ny[i];
    o.nz = r.nz[i];
    o.nl = r.nl[i];
    o.es_re = r.es_re[i];
    o.es_im = r.es_im[i];
    o.ep_re = r.ep_re[i];
    o.ep_im = r.ep_im[i];
    double k = __dmul_rn(__ddiv_rn(r.energy[i], kChbar), 1e7);
    o.k = k;
    o.kf = __ddiv_rn(k, 4.0 * kPi);
    o.pad0 = o.pad1 = o.pad2 = 0.0;
    out[i] = o;
}

struct Acc {
    double s[4];  // es_re es_im ep_re ep_im
    double c[4];  // Kahan compensators
};

__device__ __forceinline__ void kahan_add(double& sum, double& comp, double term) {
    double y = __dsub_rn(term, comp);
    double t = __dadd_rn(sum, y);
    comp = __dsub_rn(__dsub_rn(t, sum), y);
    sum = t;
}

// sin and cos of an FP64 phase x, |x| < 2^50, to about one ulp of 1.
//
// x = n pi/2 + r with n = rint(x 2/pi): fma(-n, T1, x) is x - n T1 rounded
// once (T1 = fl(pi/2); the product is exact inside the FMA and |r| < 0.8), the
// second FMA subtracts n T2 (T2 = fl(pi/2 - T1), up to 0.05 at 2^50), and the
// neglected third part is below 2e-18, so r carries at most two roundings of
// 2^-54. sin and cos of |r| <= pi/4 are r + r^3 S(r^2) and
// 1 - r^2/2 + r^4 C(r^2), S and C of degree 5 interpolated at the Chebyshev
// nodes of [0, (pi/4)^2] from their power series in 60-digit arithmetic
// (largest error 1.5e-17 and 1e-18). The quadrant n mod 4 swaps and negates.
__device__ __forceinline__ void sincos_quadrant(double x, double* sn, double* cs) {
    constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer
    const double t = fma(x, 0.6366197723675814, kMagic);
    const int q = __double2loint(t);  // n mod 2^32
    const double n = t - kMagic;
    double r = fma(-n, 1.5707963267948966, x);
    r = fma(-n, 6.123233995736766e-17, r);
    const double z = r * r;
    double s = fma(z, 1.5918129014234338e-10, -2.5051131841108444e-08);
    double c = fma(z, -1.1382632249960623e-11, 2.0876146265966424e-09);
    s = fma(z, s, 2.755731610253375e-06);
    c = fma(z, c, -2.75573172717181e-07);
    s = fma(z, s, -0.00019841269836758538);
    c = fma(z, c, 2.4801587298765665e-05);
    s = fma(z, s, 0.008333333333330948);
    c = fma(z, c, -0.0013888888888887398);
    s = fma(z, s, -0.16666666666666666);
    c = fma(z, c, 0.041666666666666664);
    s = fma(r * z, s, r);
    c = fma(z, fma(z, c, -0.5), 1.0);
    const bool swap = q & 1;
    const double a = swap ? c : s, b = swap ? s : c;
    // sin is negative in quadrants 2 and 3, cos in 1 and 2.
    *sn = __hiloint2double(__double2hiint(a) ^ ((q & 2) << 30), __double2loint(a));
    *cs = __hiloint2double(__double2hiint(b) ^ (((q + 1) & 2) << 30), __double2loint(b));
}

// path = sqrt(p2) and 1/path. A reciprocal square root seed (relative error e
// below 2^-20) takes one third-order step, y (1 + e/2 + 3 e^2/8) (Halley), and
// the square root p2 y its residual correction (Markstein): the residual
// p2 - g^2 is exact in an FMA, so g + residual y / 2 rounds as the exact root
// does. The phase k path needs that (one ulp of a 1 m path is 6e-6 rad at
// 10 keV); a division per quotient does not, so both quotients by the path
// multiply by the reciprocal instead.
__device__ __forceinline__ double sqrt_and_rcp(double p2, double* inv) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(p2));
    const double e = fma(-(p2 * y), y, 1.0);
    y = fma(y * e, fma(0.375, e, 0.5), y);
    double g = p2 * y;
    g = fma(fma(-g, g, p2), 0.5 * y, g);
    *inv = fma(y, fma(-g, y, 1.0), y);
    return g;
}

// Whatever the fast form does not take: the library functions.
__device__ __noinline__ void geometry_general(double p2, double k, double* path, double* inv,
                                              double* s, double* c) {
    *path = __dsqrt_rn(p2);
    *inv = __ddiv_rn(1.0, *path);
    sincos(__dmul_rn(k, *path), s, c);
}

// One ray against PPT screen points. The points' chains are independent, so
// they are evaluated side by side and share the ray's values and the
// polynomials' constants.
template <int PPT>
__device__ __forceinline__ void pairs_f64(const RayRec64& r, const double (&px)[PPT],
                                          const double (&py)[PPT], const double (&pz)[PPT],
                                          Acc (&acc)[PPT]) {
    double p2[PPT], nd[PPT], inv[PPT], phase[PPT], s[PPT], c[PPT];
    bool fast = true;
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
        const double dx = __dsub_rn(px[i], r.x);
        const double dy = __dsub_rn(py[i], r.y);
        const double dz = __dsub_rn(pz[i], r.z);
        // Rounded as the reference rounds it: the phase is k times the root.
        p2[i] = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
        nd[i] = fma(r.nz, dz, fma(r.ny, dy, r.nx * dx));
        phase[i] = __dmul_rn(r.k, sqrt_and_rcp(p2[i], &inv[i]));
        // 2^-198 <= p2 < 2^817 (path > 1e-30, no under- or overflow above)
        // and |phase| < 2^50; NaN and infinities fall outside.
        fast = fast &&
               (unsigned)(__double2hiint(p2[i]) - 0x33900000) < 0x73000000u - 0x33900000u &&
               (__double2hiint(phase[i]) & 0x7fffffff) < 0x43100000;
    }
    bool skip[PPT] = {};
    if (fast) {
#pragma unroll
        for (int i = 0; i < PPT; ++i) sincos_quadrant(phase[i], &s[i], &c[i]);
    } else {
#pragma unroll
        for (int i = 0; i < PPT; ++i) {
            double path;
            geometry_general(p2[i], r.k, &path, &inv[i], &s[i], &c[i]);
            skip[i] = path < 1e-30;  // diffraction.rs:81
        }
    }
#pragma unroll
    for (int i = 0; i < PPT; ++i) {
        if (skip[i]) continue;
        const double af = r.kf * fma(nd[i], inv[i], r.nl) * inv[i];
        // u = i*af*exp(i*phase) = (-af*sin, af*cos)  (diffraction.rs:98)
        const double us = af * s[i], uc = af * c[i];
        Acc& a = acc[i];
        kahan_add(a.s[0], a.c[0], fma(-r.es_re, us, -(r.es_im * uc)));
        kahan_add(a.s[1], a.c[1], fma(r.es_re, uc, -(r.es_im * us)));
        kahan_add(a.s[2], a.c[2], fma(-r.ep_re, us, -(r.ep_im * uc)));
        kahan_add(a.s[3], a.c[3], fma(r.ep_re, uc, -(r.ep_im * us)));
    }
}

// Two points per thread at four CTAs per SM: 5.91 ms on 2^16 rays x 128^2
// points (6.00 at six CTAs, 5.88 with three points, 5.96 and 6.56 with four
// points at three and two CTAs; three or four points leave more of the last
// CTA idle on small screens).
__global__ void __launch_bounds__(kF64Threads, kF64Ctas)
f64_pairs_kernel(const RayRec64* __restrict__ rays, size_t n_rays, size_t rays_per_split,
                 PixDev pix, size_t n_pix, FieldDev out, double* __restrict__ partials) {
    __shared__ RayRec64 sm[kF64Stage];
    const size_t split = blockIdx.y;
    const size_t r_begin = split * rays_per_split;
    const size_t r_end = min(n_rays, r_begin + rays_per_split);

    double px[kF64Ppt], py[kF64Ppt], pz[kF64Ppt];
    size_t pidx[kF64Ppt];
    Acc acc[kF64Ppt];
#pragma unroll
    for (int i = 0; i < kF64Ppt; ++i) {
        size_t p = blockIdx.x * (size_t)(kF64Threads * kF64Ppt) + threadIdx.x + i * kF64Threads;
        pidx[i] = p;
        size_t q = p < n_pix ? p : n_pix - 1;
        px[i] = pix.x[q];
        py[i] = pix.y[q];
        pz[i] = pix.z[q];
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[i].s[c] = acc[i].c[c] = 0.0;
    }

    for (size_t r0 = r_begin; r0 < r_end; r0 += kF64Stage) {
        const int cnt = (int)min((size_t)kF64Stage, r_end - r0);
        __syncthreads();
        const double* src = reinterpret_cast<const double*>(rays + r0);
        double* dst = reinterpret_cast<double*>(sm);
        for (int t = threadIdx.x; t < cnt * kRecDoubles; t += kF64Threads) dst[t] = src[t];
        __syncthreads();
#pragma unroll 1
        for (int j = 0; j < cnt; ++j) pairs_f64<kF64Ppt>(sm[j], px, py, pz, acc);
    }

#pragma unroll
    for (int i = 0; i < kF64Ppt; ++i) {
        size_t p = pidx[i];
        if (p >= n_pix) continue;
        if (partials == nullptr) {
            out.es_re[p] = acc[i].s[0];
            out.es_im[p] = acc[i].s[1];
            out.ep_re[p] = acc[i].s[2];
            out.ep_im[p] = acc[i].s[3];
        } else {
            // The compensated value of a Kahan accumulator is sum - comp.
            double* base = partials + split * 4 * n_pix;
#pragma unroll
            for (int c = 0; c < 4; ++c) base[c * n_pix + p] = __dsub_rn(acc[i].s[c], acc[i].c[c]);
        }
    }
}

// Adds the per-range partials of every screen point in range order, one
// thread per (point, component). The Kahan chain is serial but the loads are
// not: eight ranges are in flight while the previous eight are added.
__global__ void f64_combine_kernel(const double* __restrict__ partials, int splits, size_t n_pix,
                                   FieldDev out) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const size_t total = 4 * n_pix;
    if (i >= total) return;
    constexpr int kAhead = 8;
    double s = 0.0, c = 0.0;
    int k = 0;
    for (; k + kAhead <= splits; k += kAhead) {
        double v[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) v[u] = partials[(size_t)(k + u) * total + i];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) kahan_add(s, c, v[u]);
    }
    for (; k < splits; ++k) kahan_add(s, c, partials[(size_t)k * total + i]);
    const int comp = (int)(i / n_pix);
    double* const dst = comp == 0 ? out.es_re : comp == 1 ? out.es_im
                                              : comp == 2 ? out.ep_re : out.ep_im;
    dst[i - comp * n_pix] = s;
}

__global__ void zero_field_kernel(FieldDev out, size_t n_pix) {
    size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (p >= n_pix) return;
    out.es_re[p] = 0.0;
    out.es_im[p] = 0.0;
    out.ep_re[p] = 0.0;
    out.ep_im[p] = 0.0;
}

}  // namespace

size_t f64_splits(size_t n_rays, size_t n_pix, int num_sms, size_t* rays_per_split) {
    const size_t pix_per_cta = (size_t)kF64Threads * kF64Ppt;
    const size_t pix_ctas = (n_pix + pix_per_cta - 1) / pix_per_cta;
    // Aim for about 32 CTAs per SM in flight; never split below one stage.
    const size_t want = (size_t)num_sms * 32;
    size_t splits = (want + pix_ctas - 1) / pix_ctas;
    size_t max_splits = (n_rays + kF64Stage - 1) / kF64Stage;
    if (splits > max_splits) splits = max_splits;
    if (splits > 65535) splits = 65535;
    if (splits < 1) splits = 1;
    size_t per = (n_rays + splits - 1) / splits;
    per = (per + kF64Stage - 1) / kF64Stage * kF64Stage;
    if (rays_per_split) *rays_per_split = per;
    return per ? (n_rays + per - 1) / per : 1;
}

Status f64_reserve(size_t n_rays, size_t n_pix, int num_sms, F64Workspace& ws) {
    if (n_rays == 0 || n_pix == 0) return Status::Ok();
    XK_TRY(ws.rays.ensure(n_rays * sizeof(RayRec64)));
    const size_t splits = f64_splits(n_rays, n_pix, num_sms, nullptr);
    if (splits > 1) XK_TRY(ws.partials.ensure(splits * 4 * n_pix * sizeof(double)));
    return Status::Ok();
}

Status f64_enqueue(const RaysDev& rays, size_t n_rays, const PixDev& pix, size_t n_pix,
                   const FieldDev& out, F64Workspace& ws, cudaStream_t stream, int num_sms,
                   LaunchReport* rep) {
    if (n_pix == 0) return Status::Ok();
    if (n_rays == 0) {
        zero_field_kernel<<<(unsigned)((n_pix + 255) / 256), 256, 0, stream>>>(out, n_pix);
        XK_CUDA_TRY(cudaGetLastError());
        if (rep) rep->kernels += 1;
        return Status::Ok();
    }
    XK_TRY(ws.rays.ensure(n_rays * sizeof(RayRec64)));
    RayRec64* packed = ws.rays.as<RayRec64>();
    f64_pack_kernel<<<(unsigned)((n_rays + 255) / 256), 256, 0, stream>>>(rays, n_rays, packed);
    XK_CUDA_TRY(cudaGetLastError());

    const size_t pix_per_cta = (size_t)kF64Threads * kF64Ppt;
    const size_t pix_ctas = (n_pix + pix_per_cta - 1) / pix_per_cta;
    size_t rays_per_split = 0;
    const size_t splits = f64_splits(n_rays, n_pix, num_sms, &rays_per_split);

    double* partials = nullptr;
    if (splits > 1) {
        XK_TRY(ws.partials.ensure(splits * 4 * n_pix * sizeof(double)));
        partials = ws.partials.as<double>();
    }
    dim3 grid((unsigned)pix_ctas, (unsigned)splits);
    f64_pairs_kernel<<<grid, kF64Threads, 0, stream>>>(packed, n_rays, rays_per_split, pix, n_pix,
                                                       out, partials);
    XK_CUDA_TRY(cudaGetLastError());
    int kernels = 2;
    if (splits > 1) {
        f64_combine_kernel<<<(unsigned)((4 * n_pix + 127) / 128), 128, 0, stream>>>(
            partials, (int)splits, n_pix, out);
        XK_CUDA_TRY(cudaGetLastError());
        kernels += 1;
    }
    if (rep) rep->kernels += kernels;
    return Status::Ok();
}

}  // namespace xk

// ---------------------------------------------------------------------------
// Allocation-free variant of the FP64 path.
//
// Some callers cannot let a library call cudaMalloc: applications that have
// handed all device memory to their own pool allocator, and loops that cannot
// afford cudaMalloc's implicit device-wide synchronisation and latency on
// every call. For them xk_diffraction_f64_noalloc runs the same FP64 kernels
// as XK_PATH_F64, but its scratch (the packed ray records and the split-ray
// partial sums) lives in the fixed array below instead of context buffers.
// The array is a module global: every GPU on which this library's FP64 code
// is loaded holds its kNoAllocScratchBytes until the process exits.
// ---------------------------------------------------------------------------

namespace xk {
namespace {

constexpr size_t kNoAllocMaxRays = XK_NOALLOC_MAX_RAYS;
constexpr size_t kNoAllocRayBytes = kNoAllocMaxRays * sizeof(RayRec64);  // 16 MiB
constexpr size_t kNoAllocPartialDoubles = (size_t)2 << 20;                // 16 MiB
constexpr size_t kNoAllocScratchBytes = kNoAllocRayBytes + kNoAllocPartialDoubles * sizeof(double);
static_assert(kNoAllocScratchBytes == XK_NOALLOC_SCRATCH_BYTES, "header and scratch size agree");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// Device address of g_noalloc_scratch per device, looked up with that device
// current (a host-side reference to the symbol is not a device address). The
// address belongs to the context the module was loaded into: the cache keeps
// that context's unique id and looks the address up again when the current
// context differs (after cudaDeviceReset the module is loaded anew, possibly
// elsewhere).
constexpr int kNoAllocMaxDevices = 64;
struct NoAllocSlot {
    unsigned long long ctx_id = 0;  // 0: not looked up yet
    void* addr = nullptr;
};
std::mutex g_noalloc_mu;
NoAllocSlot g_noalloc_slot[kNoAllocMaxDevices];

// cuCtxGetCurrent / cuCtxGetId, resolved through the runtime (the library does
// not link the driver library itself).
using CtxGetCurrentFn = int (*)(void** ctx);
using CtxGetIdFn = int (*)(void* ctx, unsigned long long* id);
CtxGetCurrentFn g_ctx_get_current = nullptr;
CtxGetIdFn g_ctx_get_id = nullptr;
bool g_ctx_fns_resolved = false;

// Unique id of the calling thread's current context, 0 if there is none or it
// cannot be told. Called with g_noalloc_mu held.
unsigned long long current_ctx_id() {
    if (!g_ctx_fns_resolved) {
        g_ctx_fns_resolved = true;
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_ctx_get_current = reinterpret_cast<CtxGetCurrentFn>(f);
        f = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_ctx_get_id = reinterpret_cast<CtxGetIdFn>(f);
        cudaGetLastError();
    }
    if (!g_ctx_get_current || !g_ctx_get_id) return 0;
    void* c = nullptr;
    if (g_ctx_get_current(&c) != 0 || !c) return 0;
    unsigned long long id = 0;
    if (g_ctx_get_id(c, &id) != 0) return 0;
    return id;
}

}  // namespace
}  // namespace xk

extern "C" int xk_diffraction_f64_noalloc(const xk_rays* rays, size_t n_rays,
                                          const xk_pixels* pixels, size_t n_pix, xk_field* out,
                                          void* stream) {
    using namespace xk;
    if (n_pix == 0) return XK_OK;
    if (!pixels || !pixels->x || !pixels->y || !pixels->z || !out || !out->es_re ||
        !out->es_im || !out->ep_re || !out->ep_im)
        return XK_ERR_INVALID;
    if (n_rays > 0 && (!rays || !rays->x || !rays->y || !rays->z || !rays->nx || !rays->ny ||
                       !rays->nz || !rays->nl || !rays->es_re || !rays->es_im || !rays->ep_re ||
                       !rays->ep_im || !rays->energy))
        return XK_ERR_INVALID;
    if (n_rays > kNoAllocMaxRays) return XK_ERR_BUDGET;

    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices) {
        cudaGetLastError();
        return XK_ERR_NO_DEVICE;
    }
    void* base = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mu);
        NoAllocSlot& slot = g_noalloc_slot[dev];
        const unsigned long long id = current_ctx_id();
        if (slot.ctx_id == 0 || id != slot.ctx_id) {
            // First call on this device, a thread whose context the driver
            // does not report yet, or a context created since the lookup.
            void* p = nullptr;
            if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) {
                cudaGetLastError();
                return XK_ERR_CUDA;
            }
            slot.addr = p;
            slot.ctx_id = current_ctx_id();  // the lookup made the context current
        }
        base = slot.addr;
    }
    int num_sms = 0;
    if (cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return XK_ERR_CUDA;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    FieldDev fd{out->es_re, out->es_im, out->ep_re, out->ep_im};
    PixDev pd{pixels->x, pixels->y, pixels->z};
    if (n_rays == 0) {
        zero_field_kernel<<<(unsigned)((n_pix + 255) / 256), 256, 0, s>>>(fd, n_pix);
        return cudaGetLastError() == cudaSuccess ? XK_OK : XK_ERR_CUDA;
    }
    RaysDev rd{rays->x, rays->y, rays->z, rays->nx, rays->ny, rays->nz, rays->nl,
               rays->es_re, rays->es_im, rays->ep_re, rays->ep_im, rays->energy};
    RayRec64* packed = static_cast<RayRec64*>(base);
    double* partial_area =
        reinterpret_cast<double*>(static_cast<unsigned char*>(base) + kNoAllocRayBytes);

    // Same split rule as the allocating path, capped so the partials fit the
    // fixed area; every partial is written before it is read, so the area
    // never needs clearing.
    const size_t pix_per_cta = (size_t)kF64Threads * kF64Ppt;
    const size_t pix_ctas = (n_pix + pix_per_cta - 1) / pix_per_cta;
    const size_t want = (size_t)num_sms * 32;
    size_t splits = (want + pix_ctas - 1) / pix_ctas;
    size_t max_splits = (n_rays + kF64Stage - 1) / kF64Stage;
    if (splits > max_splits) splits = max_splits;
    const size_t fit = kNoAllocPartialDoubles / (4 * n_pix);
    if (splits > fit) splits = fit;
    if (splits > 65535) splits = 65535;
    if (splits < 1) splits = 1;
    size_t rays_per_split = (n_rays + splits - 1) / splits;
    rays_per_split = (rays_per_split + kF64Stage - 1) / kF64Stage * kF64Stage;
    splits = (n_rays + rays_per_split - 1) / rays_per_split;
    double* partials = splits > 1 ? partial_area : nullptr;

    f64_pack_kernel<<<(unsigned)((n_rays + 255) / 256), 256, 0, s>>>(rd, n_rays, packed);
    if (cudaGetLastError() != cudaSuccess) return XK_ERR_CUDA;
    dim3 grid((unsigned)pix_ctas, (unsigned)splits);
    f64_pairs_kernel<<<grid, kF64Threads, 0, s>>>(packed, n_rays, rays_per_split, pd, n_pix, fd,
                                                  partials);
    if (cudaGetLastError() != cudaSuccess) return XK_ERR_CUDA;
    if (splits > 1) {
        f64_combine_kernel<<<(unsigned)((4 * n_pix + 127) / 128), 128, 0, s>>>(
            partials, (int)splits, n_pix, fd);
        if (cudaGetLastError() != cudaSuccess) return XK_ERR_CUDA;
    }
    return XK_OK;
}
