// Double-double evaluation of k |q| in turns.
#pragma once

namespace xk {

// Fractional part of (kt_hi + kt_lo) * |q| in turns, |q| = sqrt(qx^2+qy^2+qz^2),
// evaluated in double-double arithmetic (error-free products by FMA, TwoSum,
// one Newton correction of the square root). LOW: `low` is added to the
// low-order part of |q|^2 (components given as sums of two doubles).
template <bool LOW = false>
__device__ __forceinline__ double dd_turns(double kt_hi, double kt_lo, double qx, double qy,
                                           double qz, double* qn, double* inv2q,
                                           double low = 0.0) {
    const double p0 = qx * qx, p1 = qy * qy, p2 = qz * qz;
    const double e0 = fma(qx, qx, -p0), e1 = fma(qy, qy, -p1), e2 = fma(qz, qz, -p2);
    double s1 = p0 + p1;
    double b1 = s1 - p0;
    double t1 = (p0 - (s1 - b1)) + (p1 - b1);
    double s2 = s1 + p2;
    double b2 = s2 - s1;
    double t2 = (s1 - (s2 - b2)) + (p2 - b2);
    double lo = t1 + t2 + e0 + e1 + e2;
    if (LOW) lo += low;
    double hi = s2 + lo;
    lo -= hi - s2;
    const double r = sqrt(hi);
    *qn = r;
    // 1/(2r): f32 reciprocal seed and one FP64 Newton step (~1e-14 relative);
    // it scales the square root's low-order correction and is the sweep's
    // 1/(2|q|).
    const double d2 = 2.0 * r;
    const double y0 = (double)__frcp_rn((float)d2);
    const double y = fma(y0, fma(-d2, y0, 1.0), y0);
    *inv2q = y;
    const double rl = (fma(-r, r, hi) + lo) * y;
    const double ph = kt_hi * r;
    const double pe = fma(kt_hi, r, -ph) + (kt_hi * rl + kt_lo * r);
    return (ph - rint(ph)) + pe;
}

// a - b as an unevaluated sum (Knuth's two-difference).
__device__ __forceinline__ double dd_diff(double a, double b, double* lo) {
    const double d = a - b;
    const double bb = d - a;
    *lo = (a - (d - bb)) - (b + bb);
    return d;
}

}  // namespace xk
