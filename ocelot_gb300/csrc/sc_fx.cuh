// Block fixed point for the FP64 form's transforms: the values of one line as
// 64-bit integers under one exponent.
//
// Why: this GPU issues an FP64 instruction of a warp in 18 to 20 cycles of an SM
// (two lanes a cycle), while a 64-bit integer addition is two instructions at 64
// lanes a cycle or more, and a product's upper half three wide multiplications and a
// few additions.  A 128-point line costs 50e3 SM cycles per 32 lines on the
// FP64 pipe (2200 instructions) and about 6e3 in integers, with the conversions
// to and from double another 5e3.
//
// Precision: a line is scaled so that its largest component has its leading one in
// bit 56, 57 or 58 (fx_bit; the rest up to bit 61 is room for the transform's growth),
// so every input is rounded at half a unit, 2^-57 .. 2^-59 of that power of two, and a
// product leaves out up to two units; additions are exact.  Against a double transform, whose
// every operation rounds at 2^-53 of its own result, the error in the 2-norm is the
// smaller one: 0.31 to 0.78 of it for one transform, up to 0.99 for the x pass with its
// Green product (tests/test_fixed_point_host.py: lines of every length, random, bunch
// shaped, alternating, spikes, 20 decades).  As with any FFT the error is one of the
// line's norm: a value 2^5 and more below the largest is held with less than 53 bits.
//
// A line with a NaN or an infinity comes out as NaNs (a double transform spreads
// them over the line too).
#pragma once
#include "sc_cx.cuh"

namespace ocsc {

struct Fx {
    long long v;
};
__host__ __device__ __forceinline__ Fx operator+(Fx a, Fx b) { return Fx{a.v + b.v}; }
__host__ __device__ __forceinline__ Fx operator-(Fx a, Fx b) { return Fx{a.v - b.v}; }
__host__ __device__ __forceinline__ Fx operator-(Fx a) { return Fx{-a.v}; }
__host__ __device__ __forceinline__ Fx& operator+=(Fx& a, Fx b) { a.v += b.v; return a; }
__host__ __device__ __forceinline__ Fx& operator-=(Fx& a, Fx b) { a.v -= b.v; return a; }
struct __align__(16) Fx2 {
    Fx x, y;
};
template <> struct CT<Fx> { using T = Fx2; };

// a factor |w| <= 1 as H / 2^31 + L / 2^62, 0 <= L < 2^31 (1 itself as 1 - 2^-62)
struct FxC {
    int H, L;
    __host__ __device__ constexpr FxC(int h, int l) : H(h), L(l) {}
    __host__ __device__ constexpr explicit FxC(double w) : H(0), L(0) {
        const double q = w * 4611686018427387904.0;
        const long long i = q >= 4611686018427387904.0 ? 4611686018427387903ll : (long long)q;
        H = (int)(i >> 31);
        L = (int)(i & 0x7fffffff);
    }
    __host__ __device__ constexpr FxC operator-() const { return FxC(-H, -L); }
};
// the table entry of a twiddle wr + i wi
struct __align__(16) FxW {
    FxC r, i;
};

__host__ __device__ __forceinline__ int fx_hi(Fx a) { return (int)(a.v >> 32); }
__host__ __device__ __forceinline__ int fx_lo(Fx a) { return (int)((unsigned)a.v >> 1); }

// a w, |a| < 2^62: the 64-bit operand as its high word and 31 bits of its low one
// (the product of the low parts, up to two units, and the low bit are left out)
__host__ __device__ __forceinline__ Fx fx_mul(Fx a, FxC w, long long half = 1ll << 29) {
    const int ah = fx_hi(a), al = fx_lo(a);
    long long m = half + (long long)ah * w.L;
    m += (long long)al * w.H;
    const long long h = (long long)ah * w.H;
    return Fx{h + h + (m >> 30)};
}
// the same for a compile-time constant, with the mean of what is left out in the
// rounding, as far as 0 still gives 0: a DFT sums the products of one constant, and
// their common bias with them (256-point pass over one spike: 1.14 -> 0.99 of a
// double pass's error)
__host__ __device__ __forceinline__ Fx fx_mul_const(Fx a, FxC w) {
    const long long half = (1ll << 29) + w.L / 2 + w.H / 4;
    return fx_mul(a, w, half < 0 ? 0 : half > (1ll << 30) - 1 ? (1ll << 30) - 1 : half);
}
// a u + b w for |a|, |b| < 2^61 and u^2 + w^2 <= 1: the middle sum stays below 1.92 * 2^62
__host__ __device__ __forceinline__ Fx fx_mul2(Fx a, FxC u, Fx b, FxC w) {
    const int ah = fx_hi(a), al = fx_lo(a), bh = fx_hi(b), bl = fx_lo(b);
    long long m = (1ll << 29) + (long long)ah * u.L;
    m += (long long)al * u.H;
    m += (long long)bh * w.L;
    m += (long long)bl * w.H;
    long long h = (long long)ah * u.H;
    h += (long long)bh * w.H;
    return Fx{h + h + (m >> 30)};
}

// the bit of the largest input's leading one, so that a DFT over n inputs
// stays below 2^61.5: each output is at most n sqrt(2) 2^(bit + 1)
__host__ __device__ constexpr int fx_bit(int n) {
    int lg = 0;
    while ((1 << lg) < n) ++lg;
    return 60 - lg;
}
// magnitude of a value for a maximum: its high word's (+ 1 for negative ones)
__host__ __device__ __forceinline__ unsigned fx_mag(Fx a) {
    const int h = fx_hi(a);
    return (unsigned)(h < 0 ? ~h : h);
}
// bits to shift out before an n-point DFT of values of magnitudes up to mag
template <int N>
__device__ __forceinline__ int fx_room(unsigned mag) {
    const int bits = 64 - __clz((int)mag);  // |value| < 2^bits
    const int s = bits - (fx_bit(N) + 1);
    return s > 0 ? s : 0;
}
// a / 2^s rounded, 0 <= s < 32
__host__ __device__ __forceinline__ Fx fx_down(Fx a, int s) {
    return Fx{(a.v + ((1ll << s) >> 1)) >> s};
}
__host__ __device__ __forceinline__ Fx2 fx_down(Fx2 a, int s) { return Fx2{fx_down(a.x, s), fx_down(a.y, s)}; }

constexpr int FX_BAD = 0x7ff;  // the line exponent of a NaN or an infinity

// biased exponent bits of a double (0 for zeros and denormals)
__device__ __forceinline__ int fx_exp(double d) { return (__double2hiint(d) >> 20) & 0x7ff; }

// shifts by 0 and more that give 0 (arithmetic: the sign) for 64 and more
__device__ __forceinline__ unsigned long long fx_shr(unsigned long long m, int s) {
#ifdef __CUDA_ARCH__
    unsigned long long r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(m), "r"(s));
    return r;
#else
    return s > 63 ? 0 : m >> s;
#endif
}
__device__ __forceinline__ long long fx_sar(long long v, int s) {
#ifdef __CUDA_ARCH__
    long long r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
    return r;
#else
    return v >> (s > 63 ? 63 : s);
#endif
}
__device__ __forceinline__ long long fx_shl(long long v, int s) {
#ifdef __CUDA_ARCH__
    long long r;
    asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
    return r;
#else
    return s > 63 ? 0 : (long long)((unsigned long long)v << s);
#endif
}
// a / 2^s rounded, or a 2^-s for a negative s; |a| < 2^62, and the result's as well
__device__ __forceinline__ Fx fx_scale(Fx a, int s) {
    const int right = max(s, 0);
    return Fx{fx_shl(fx_sar(a.v + (fx_shl(1ll, right) >> 1), right), max(-s, 0))};
}
__device__ __forceinline__ Fx2 fx_scale(Fx2 a, int s) { return Fx2{fx_scale(a.x, s), fx_scale(a.y, s)}; }

// a double factor as w 2^(e - 1022), 1/2 <= |w| < 1 with all its bits
__device__ __forceinline__ FxC fx_fraction(double g, int& e) {
    const int hi = __double2hiint(g), sg = hi >> 31;
    const unsigned lo = (unsigned)__double2loint(g);
    e = fx_exp(g);
    const int H = (int)(((unsigned)hi & 0xfffffu) << 10 | lo >> 22) | (e ? 0x40000000 : 0);
    const int L = (int)((lo & 0x3fffffu) << 9);
    e = max(e, 1);
    return FxC((H ^ sg) - sg, (L ^ sg) - sg);
}
// a bound on the leading bit of a value under that exponent; above any of a
// finite one where the factor is a NaN or an infinity
__device__ __forceinline__ int fx_top(Fx2 a, int e) {
    return e == FX_BAD ? 1 << 20 : 64 - __clz((int)max(fx_mag(a.x), fx_mag(a.y))) + e;
}

// d as an integer of a line of exponent E >= fx_exp(d), E >= 1: a value with exponent E
// has bit B as its leading one
template <int B>
__device__ __forceinline__ Fx fx_from(double d, int E) {
    const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
    const int e = (hi >> 20) & 0x7ff;
    const unsigned long long m =
        ((unsigned long long)(hi << 11 | lo >> 21 | (e ? 0x80000000u : 0u)) << 32) | (lo << 11);
    const int s = E - max(e, 1) + (62 - B);
    const long long r = (long long)((fx_shr(m, s) + 1) >> 1);
    const long long sg = (int)hi >> 31;
    return Fx{(r ^ sg) - sg};
}

// what fx_to needs of a line of exponent E with bit B for 2^E
struct FxOut {
    int ebase, ezero, ovf;
    __device__ __forceinline__ FxOut(int E, int B) {
        const bool bad = E == FX_BAD;
        ebase = bad ? 1 << 20 : E - B + 63;
        ezero = bad ? 1 << 20 : 0;
        ovf = bad ? 0x7ff80000 : 0x7ff00000;
    }
};
// the nearest double (below the normal range the nearest denormal)
__device__ __forceinline__ double fx_to(Fx a, FxOut o) {
    const long long sg = a.v >> 63;
    const unsigned long long u = (unsigned long long)((a.v ^ sg) - sg);
    const int n = __clzll((long long)u);
    const unsigned long long w = u << (n & 63);
    const int e = u ? o.ebase - n : o.ezero, en = max(e, 1);
    const unsigned long long m = (fx_shr(w, 10 + en - e) + 1) >> 1;
    unsigned hi = (unsigned)(m >> 32) + ((unsigned)(en - 1) << 20), lo = (unsigned)m;
    if (e > 2046) {
        hi = (unsigned)o.ovf;
        lo = 0;
    }
    return __hiloint2double((int)(hi | ((unsigned)sg & 0x80000000u)), (int)lo);
}

// the nearest double of a 2^-S
template <int S = 0>
__device__ __forceinline__ double fx_double(Fx a) {
    const long long sg = a.v >> 63;
    const unsigned long long u = (unsigned long long)((a.v ^ sg) - sg);
    const int n = __clzll((long long)u);
    const unsigned long long m = (((u << (n & 63)) >> 10) + 1) >> 1;
    const unsigned hi = (unsigned)(m >> 32) + ((unsigned)(1085 - S - n) << 20) | ((unsigned)sg & 0x80000000u);
    return u ? __hiloint2double((int)hi, (int)(unsigned)m) : 0.0;
}

// Field grids of the FP64 kick: differences of the potential as integers whose
// bit FX_PHI stands for 2^(the largest exponent of the potential)
constexpr int FX_PHI = 58;

}  // namespace ocsc
