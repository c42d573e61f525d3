// FP64 square root, quotient, logarithm and arctangent for the exact integrated
// Green's function (igf_point in sc_green.cu).  That table is bound by the FP64
// pipe (about 1/64 of the FP32 rate on this GPU), so the square root, the
// quotients and the reference's own products and sums are FP64 and everything else
// runs on the integer pipes beside them: table-driven reductions in the manner
// of P. T. P. Tang (ACM TOMS 16, 1990), the remaining series in 64-bit integers,
// its terms below 2^-26 (log) and 2^-34 (atan) in FP32.  Results are
// within 0.50 (sqrt), 0.80 (log; 0.51 for |log x| > 1, the most just beyond |x - 1| = 2^-8)
// and 1.09 (atan of a quotient; 1.45 where it lies just below a power of two and the
// quotient above) ulp of the exact value over the arguments tried (millions each against
// 113-bit arithmetic).
// FP64 instructions: sqrt 7, log none, atan of a quotient 7 (10 and 20 in a form
// with its series in FP64: 63^3 beside the other stream 75 -> 46 us at 10k
// particles, 84 -> 54 at 200k; 48 and 56 since the logarithm keeps its accuracy near 1).
//
// Arguments must be positive and inside 2^+-180 (igf_regular checks the mesh steps
// once; others take the CUDA functions, igf_point).
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

constexpr long long LN2_HI = 49946518145322873ll;  // ln 2 in units of 2^-56
constexpr long long LN2_LO = 2882134964ll;  // and the rest of it in units of 2^-88

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
// FP32 -> FP64 on the integer pipes (the conversions issue on the FP64 pipe):
// exact, subnormals 0
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

// upper half of a product
SC_HD long long mulhi(long long a, long long b) {
#ifdef __CUDA_ARCH__
    return __mul64hi(a, b);
#else
    return (long long)(((__int128)a * b) >> 64);
#endif
}
SC_HD int clz64(unsigned long long v) {
#ifdef __CUDA_ARCH__
    return __clzll((long long)v);
#else
    return v ? __builtin_clzll(v) : 64;
#endif
}
SC_HD unsigned long long shr64(unsigned long long v, int n) {  // 0 for n > 63
#ifdef __CUDA_ARCH__
    unsigned long long r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
    return r;
#else
    return n > 63 ? 0 : v >> n;
#endif
}
// the nearest double of v 2^-s
SC_HD double to_double(long long v, int s) {
    const long long sg = v >> 63;
    const unsigned long long u = (unsigned long long)((v ^ sg) - sg);
    const int n = clz64(u);
    const unsigned long long m = (((u << (n & 63)) >> 10) + 1) >> 1;
    const unsigned hi = ((unsigned)(m >> 32) + ((unsigned)(1085 - n - s) << 20)) | ((unsigned)sg & 0x80000000u);
    return u ? bits_d(hi, (unsigned)m) : 0.0;
}

// log(x) for normal x > 0: x = 2^k m, m in [1, 2); with the table's short 1/c
// near 1/m, r = m (1/c) - 1, exact in units of 2^-66, |r| < 2^-7.9, and
// log x = k ln2 - log(1/c) + r - r^2 (1/2 - r/3 + r^2/4 - [r^3/5 - r^4/6 + r^5/7 - r^6/8 in FP32]),
// in integers; the sum in units of 2^-56, 2^-58 or 2^-62, the finer ones for the smaller
// results.  1 - 2^-8 <= x < 1 + 2^-8, where the result may be of any size, takes 1/c = 1: log x = r (1 - r (1/2 - ...)), r with all its bits.
SC_HD double log_(double x, const LogEntry* __restrict__ tab) {
    const unsigned hx = hi_d(x);
    const int k = (int)(hx >> 20) - 1023;
    const LogEntry t = tab[(hx >> 13) & 127u];
    const bool near1 = hx - 0x3fefe000u < 0x3000u;  // 1 - 2^-8 <= x < 1 + 2^-8: k is -1 or 0
    const unsigned ic = near1 ? (1u << 14) >> (k & 1) : (unsigned)t.ic;
    const unsigned long long m = ((unsigned long long)((hx & 0xfffffu) | 0x100000u) << 32) | lo_d(x);
    const long long r = (long long)(m * (unsigned long long)ic);  // 2^-66; the 1 is 2^66, gone
    const long long r4 = (long long)((unsigned long long)r << 4);
    const long long r2 = mulhi(r4, r4);                           // 2^-76
    const float rf = (float)(int)(r >> 32) * 0x1p-34f;
    const float f = (rf * rf) * rf * fmaf(rf, fmaf(rf, fmaf(rf, -0.125f, 0.142857143f), -0.166666667f), 0.2f);
    const long long u = (1ll << 61) - (mulhi(r, 0x5555555555555555ll) >> 4) + (r2 >> 16) -
                        (long long)((unsigned long long)(long long)(int)(f * 0x1p50f) << 12);  // 2^-62
    const long long q = r - (mulhi(r2, u) >> 8);                                     // 2^-66
    const long long low = (((long long)k * LN2_LO + (1 << 25)) >> 26) + t.t + ((q + 8) >> 4);  // 2^-62
    // bits more than 2^-56: |log x| < 2 for k = -2 .. 1, < 2^5 for -40 .. 40
    const int sh = (unsigned)(k + 2) <= 3u ? 6 : ((unsigned)(k + 40) <= 80u ? 2 : 0);
    long long v = (long long)((unsigned long long)((long long)k * LN2_HI) << sh) + ((low + (32 >> sh)) >> (6 - sh));
    int s = 56 + sh;
    if (near1) {
        const long long sg = r >> 63;
        const unsigned long long ur = (unsigned long long)((r ^ sg) - sg);
        const int n = clz64(ur);                                 // 5 and more
        const long long rn = (long long)(ur << ((n - 1) & 63));  // |r| 2^(65 + n)
        v = (mulhi(rn, (1ll << 62) - ((mulhi(r4, u) + 32) >> 6)) ^ sg) - sg;
        s = 63 + n;
    }
    return to_double(v, s);
}

// w = |n| / |d| to FP32 accuracy, 2^-30 .. 2^30 (n, d normal)
SC_HD float ratio(double n, double d) {
    const unsigned hn = hi_d(n), hd = hi_d(d);
    const float fn = f_bits(((hn & 0xfffffu) << 3) | (lo_d(n) >> 29) | 0x3f800000u);
    const float fd = f_bits(((hd & 0xfffffu) << 3) | (lo_d(d) >> 29) | 0x3f800000u);
    int e = (int)((hn >> 20) & 0x7ffu) - (int)((hd >> 20) & 0x7ffu);
    e = e < -30 ? -30 : (e > 30 ? 30 : e);
    return fn / fd * f_bits((unsigned)(127 + e) << 23);
}
// atan(n / d), any signs: with w = |n / d|, w <= 1 about c = j/128 as atan c + atan((n - c d) / (d + c n)),
// w > 1 about 1/c as pi/2 - atan c + atan((c n - d) / (n + c d)), w < 3.5/128 as itself: one quotient t,
// |t| <= 2^-8, and w itself never rounded; t in FP64, t - t (t^2/3 - t^4/5 + [t^6/7 - t^8/9 + t^10/11 in FP32]) and
// the sum in integers, in units that leave the result 59 bits or more
SC_HD double atan_(double n, double d, const AtanEntry* __restrict__ tab) {
    const unsigned sign = (hi_d(n) ^ hi_d(d)) & 0x80000000u;
    const double an = bits_d(hi_d(n) & 0x7fffffffu, lo_d(n)), ad = bits_d(hi_d(d) & 0x7fffffffu, lo_d(d));
    const float af = ratio(an, ad);
    const bool big = af > 1.0f;
    const float u = big ? 1.0f / af : af;
    int j = (int)(u * 128.0f + 0.5f);  // 0 .. 128
    const bool tiny = !big && j < 4;   // the quotient's rounding would be the result's
    if (tiny) j = 0;
    const float cf = (float)j * 0.0078125f;
    const double c = widen(cf);
    const double p = big ? ad : an, q = big ? an : ad;  // p <= q
    const double N = fma(-c, q, p), D = fma(c, p, q);
    const double t = div_(big ? bits_d(hi_d(N) ^ 0x80000000u, lo_d(N)) : N, D);
    const AtanEntry E = tab[j];
    const unsigned ht = hi_d(t);
    const int e = (int)((ht >> 20) & 0x7ffu) - 1023;
    const unsigned long long m = (((unsigned long long)((ht & 0xfffffu) | 0x100000u) << 32) | lo_d(t)) << 9;  // |t| 2^(61 - e)
    const long long tq = (long long)shr64(m, -5 - e);  // 2^-66
    const long long t2 = mulhi(tq, tq);                // 2^-68
    const long long t4 = mulhi(t2 << 5, t2 << 5);      // 2^-82
    const float t2f = (float)(int)(t2 >> 32) * 0x1p-36f;
    const float f = (t2f * t2f) * t2f * fmaf(t2f, fmaf(t2f, 0.0909090909f, -0.111111111f), 0.142857143f);
    const long long corr = mulhi(t2, 0x5555555555555555ll) - (mulhi(t4, 0x3333333333333333ll) >> 14) +
                           ((long long)(int)(f * 0x1p64f) << 4);  // 2^-68
    const int s = tiny ? 61 - e : (big ? 61 : E.s);
    const long long T = (long long)shr64(m, 61 - e - s);
    const long long ti = T - (mulhi(T, corr << 6) >> 10);
    const long long v = tiny ? ti : (big ? E.hi2 : E.hi) + ((int)ht < 0 ? -ti : ti);
    const double res = tiny && e < -1000 ? t : to_double(v, s);
    return bits_d(hi_d(res) ^ sign, lo_d(res));
}

// IG of sc.py:109-133 at one corner: the reference's operations, the four
// functions above in the place of numpy's (the products with -1/2 are exact)
SC_HD double point_(double x, double y, double z, const LogEntry* __restrict__ lt, const AtanEntry* __restrict__ at) {
    const double x2 = x * x, y2 = y * y, z2 = z * z;
    const double r = sqrt_((x2 + y2) + z2);
    const double yz = y * z, zx = z * x, xy = x * y;
    const double t1 = (-0.5 * x2) * atan_(yz, x * r, at);
    const double t2 = yz * log_(x + r, lt);
    const double t3 = (0.5 * y2) * atan_(zx, y * r, at);
    const double t4 = zx * log_(y + r, lt);
    const double t5 = (0.5 * z2) * atan_(xy, z * r, at);
    const double t6 = xy * log_(z + r, lt);
    return ((((t1 + t2) - t3) + t4) - t5) + t6;
}

}  // namespace igf
}  // namespace ocsc
