// FP64 square root, quotient, logarithm and arctangent for the exact integrated
// Green's function (igf_point in sc_green.cu).  That table is bound by the FP64
// pipe (about 1/64 of the FP32 rate on this GPU), so these spend FP64
// instructions only where 53 bits are needed: table-driven reductions in the
// manner of P. T. P. Tang (ACM TOMS 16, 1990), the leading terms of the
// remaining series in FP64, the higher ones -- below 2^-32 of the result -- and
// every exponent and table-index step on the FP32 and integer pipes.  Results
// are within 0.51 (sqrt, quotient) and 0.53 (log, atan) ulp of the exact value
// over the arguments tried (10 million each against extended precision).
// Instructions: sqrt 7, quotient 5, log 10, atan 15.
//
// Arguments must be positive and well inside the exponent range (igf_point
// checks the mesh steps once and falls back to the CUDA functions).
#pragma once
#include <string.h>

#include "sc_igf_tables.cuh"

#ifdef __CUDA_ARCH__
#define SC_HD __device__ __forceinline__
#else
#define SC_HD static inline
#endif

namespace ocsc {
namespace igf {

SC_HD double bits_d(unsigned hi, unsigned lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    const unsigned long long u = ((unsigned long long)hi << 32) | lo;
    double d;
    memcpy(&d, &u, 8);
    return d;
#endif
}
SC_HD unsigned hi_d(double d) {
#ifdef __CUDA_ARCH__
    return (unsigned)__double2hiint(d);
#else
    unsigned long long u;
    memcpy(&u, &d, 8);
    return (unsigned)(u >> 32);
#endif
}
SC_HD unsigned lo_d(double d) {
#ifdef __CUDA_ARCH__
    return (unsigned)__double2loint(d);
#else
    unsigned long long u;
    memcpy(&u, &d, 8);
    return (unsigned)u;
#endif
}
SC_HD unsigned bits_f(float f) {
    unsigned u;
    memcpy(&u, &f, 4);
    return u;
}
SC_HD float f_bits(unsigned u) {
    float f;
    memcpy(&f, &u, 4);
    return f;
}
// FP64 <-> FP32 on the integer pipes (the conversions issue on the FP64 pipe):
// rounded half up to FP32, below FP32's normal range 0; widened exactly, subnormals 0
SC_HD float narrow(double d) {
    const unsigned hi = hi_d(d), mag = hi & 0x7fffffffu;
    if (mag < (897u << 20)) return 0.0f;
    if (mag >= (1150u << 20)) return f_bits((hi & 0x80000000u) | 0x7f7fffffu);
    return f_bits((hi & 0x80000000u) | (((mag << 3) | (lo_d(d) >> 29)) - (896u << 23) + ((lo_d(d) >> 28) & 1u)));
}
SC_HD double widen(float f) {
    const unsigned u = bits_f(f), m = u & 0x7fffffffu;
    if (m < 0x00800000u) return bits_d(u & 0x80000000u, 0u);
    return bits_d((u & 0x80000000u) | ((m >> 3) + 0x38000000u), u << 29);
}
// starting values to ~20 bits or better
SC_HD double rcp_start(double x) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
#else
    return bits_d(hi_d(1.0 / x), 0u);
#endif
}
SC_HD double rsqrt_start(double x) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
#else
    return bits_d(hi_d(1.0 / sqrt(x)), 0u);
#endif
}

// sqrt(x): Goldschmidt's iteration and a residual correction
SC_HD double sqrt_(double x) {
    const double y = rsqrt_start(x);
    double g = x * y, h = 0.5 * y;
    const double r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    return fma(fma(-g, g, x), h, g);
}
// n / d: one Newton-Raphson step on 1/d, the quotient and its residual
SC_HD double div_(double n, double d) {
    double y = rcp_start(d);
    y = fma(y, fma(-d, y, 1.0), y);
    const double q = n * y;
    return fma(fma(-q, d, n), y, q);
}

// log(x) for normal x > 0: x = 2^k m, m in [1, 2); with the table's short 1/c
// near 1/m, r = m (1/c) - 1 (exact up to 2^-62), |r| < 2^-7.9, and
// log x = (k ln2_hi + hi) + r - r^2/2 + r^3/3 + [r^4 (..) + k ln2_lo + lo in FP32]
SC_HD double log_(double x, const LogEntry* __restrict__ tab) {
    const unsigned hx = hi_d(x);
    const float k = (float)((int)(hx >> 20) - 1023);
    const LogEntry t = tab[(hx >> 13) & 127u];
    const double m = bits_d((hx & 0xfffffu) | 0x3ff00000u, lo_d(x));
    const double r = fma(m, widen(t.invc), -1.0);
    const double hi = fma(widen(k), 0x1.62e42fefa3800p-1, t.hi);  // exact: both multiples of 2^-42
    const double w = hi + r, e = (hi - w) + r;
    const float rf = narrow(r), r2f = rf * rf;
    const float s = fmaf(rf, fmaf(rf, fmaf(rf, 0.142857143f, -0.166666667f), 0.2f), -0.25f);
    const float tail = fmaf(r2f * r2f, s, fmaf(k, 0x1.ef357ap-45f, t.lo));
    const double q = fma(r, 0x1.5555555555555p-2, -0.5);
    return w + (fma(r * r, q, widen(tail)) + e);
}

// atan(w), any sign of a finite w: |w| <= 1 about c = j/128 as atan c + atan((w - c) / (1 + c w)),
// |w| > 1 about 1/c as pi/2 - atan c + atan((c w - 1) / (w + c)); the quotient t, |t| <= 2^-8, and
// t - t^3/3 in FP64, the rest of the series in FP32
SC_HD double atan_(double w, const AtanEntry* __restrict__ tab) {
    const unsigned sign = hi_d(w) & 0x80000000u;
    const double a = bits_d(hi_d(w) & 0x7fffffffu, lo_d(w));
    const bool big = hi_d(a) >= 0x3ff00000u;  // |w| >= 1
    const float af = narrow(a);
    const float u = big ? 1.0f / af : af;
    const int j = (int)(u * 128.0f + 0.5f);  // 0 .. 128
    const float cf = (float)j * 0.0078125f;
    const double c = widen(cf), mc = widen(-cf);
    // N = w - c, D = 1 + c w, or N = c w - 1, D = w + c
    const double N = fma(big ? c : 1.0, a, big ? -1.0 : mc);
    const double D = fma(big ? 1.0 : c, a, big ? c : 1.0);
    const double t = div_(N, D);
    const double hi = big ? tab[j].hi2 : tab[j].hi;
    const float lo = big ? tab[j].lo2 : tab[j].lo;
    const float tf = narrow(t), t2f = tf * tf;
    const float tail = fmaf(tf * (t2f * t2f), fmaf(t2f, -0.142857143f, 0.2f), lo);
    const double t3 = (t * t) * t;
    const double corr = fma(t3, -0x1.5555555555555p-2, widen(tail));
    const double s = hi + t, e = (hi - s) + t;
    const double v = s + (e + corr);
    return bits_d(hi_d(v) ^ sign, lo_d(v));
}

// IG of sc.py:109-133 at one corner: the reference's operations, the four
// functions above in the place of numpy's (the products with -1/2 are exact)
SC_HD double point_(double x, double y, double z, const LogEntry* __restrict__ lt, const AtanEntry* __restrict__ at) {
    const double x2 = x * x, y2 = y * y, z2 = z * z;
    const double r = sqrt_((x2 + y2) + z2);
    const double yz = y * z, zx = z * x, xy = x * y;
    const double t1 = (-0.5 * x2) * atan_(div_(yz, x * r), at);
    const double t2 = yz * log_(x + r, lt);
    const double t3 = (0.5 * y2) * atan_(div_(zx, y * r), at);
    const double t4 = zx * log_(y + r, lt);
    const double t5 = (0.5 * z2) * atan_(div_(xy, z * r), at);
    const double t6 = xy * log_(z + r, lt);
    return ((((t1 + t2) - t3) + t4) - t5) + t6;
}

}  // namespace igf
}  // namespace ocsc
