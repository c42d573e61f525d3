// The two-step FFT's register DFTs, in FP32 and in block fixed point (and in FP64,
// which only the host test that compares the two takes).  No shared memory and no
// device state: the file compiles for the host as well.
#pragma once
#include <type_traits>

#include "sc_fx.cuh"

namespace ocsc {

// Two-step FFT (lines of length L = P * Q, P <= Q).  With n = Q n1 + n2 and
// k = k1 + P k2,
//   X[k1 + P k2] = sum_n2 w_Q^(n2 k2) w_L^(n2 k1) sum_n1 w_P^(n1 k1) x[Q n1 + n2].
// Step 1, one work item per (line, n2): the P-point DFT over n1 in registers,
// the twiddle w_L^(n2 k1), each k1 stored in row k1 of a table with rows of
// Q + 1.  Step 2, one item per (line, k1): the Q-point DFT over n2 in
// registers, stored in natural order.  Every butterfly stays in registers:
// one shared-memory round trip and one barrier per step against one per
// radix stage of the Stockham passes, and about half their instructions.
// Work items run line-fastest (LF) when a power-of-two count of 8 (FP64) or 16
// lines or more shares the block: the lanes of a quarter- or half-warp then
// hold as many lines at the same offset, which the odd line stride puts on
// distinct banks.  The twiddles come as tw2[k1 * Q + n2] = w_L^(n2 k1)
// (load_twiddles lays the table out so for these lengths).
//
// The register DFTs count instructions: the factors of the odd half are folded
// into the final additions as fused multiply-adds (a rotation by c - i s costs
// c (1 - i s/c), two instructions, and the factor c rides on the four
// additions; Linzer and Feig's form), and HALF leaves out what the caller's
// zero padding makes trivial -- HALF_IN: the second half of the inputs is zero;
// HALF_OUT: only the first half of the outputs is wanted.  Instructions of
// dft8 / dft16: 52 / 148 in full, 36 / 104 with HALF_IN, 44 / 132 with HALF_OUT.
// The FP64 form runs the same DFTs on 64-bit integers (R = Fx), where a factor
// is applied once and the product added and subtracted.
// ---------------------------------------------------------------------------
// the constants of the register DFTs, and a constant times a value plus another
template <typename R> struct KT { using T = R; };
template <> struct KT<Fx> { using T = FxC; };
template <typename R> using Kc = typename KT<R>::T;
__device__ __forceinline__ float fmar(float k, float b, float c) { return fmaf(k, b, c); }
__device__ __forceinline__ double fmar(double k, double b, double c) { return fma(k, b, c); }
__device__ __forceinline__ Fx fmar(FxC k, Fx b, Fx c) { return fx_mul_const(b, k) + c; }
template <typename R>
__device__ __forceinline__ Cx<R> cmulc(Cx<R> v, R wr, R wi) {  // v * (wr + i wi), constant factor
    return cx<R>(fmar(v.x, wr, -(v.y * wi)), fmar(v.x, wi, v.y * wr));
}
template <typename R>
__device__ __forceinline__ Cx<Fx> cmulc(Cx<Fx> v, FxC wr, FxC wi) {
    return cx<Fx>(fx_mul2(v.x, wr, v.y, -wi), fx_mul2(v.x, wi, v.y, wr));
}

enum DftPart { DFT_FULL = 0, HALF_IN = 1, HALF_OUT = 2 };

template <typename R, bool INV, int PART>
__device__ __forceinline__ void dftp4(Cx<R>& a0, Cx<R>& a1, Cx<R>& a2, Cx<R>& a3) {
    if constexpr (PART == HALF_IN) {  // a2 = a3 = 0
        const Cx<R> t = INV ? cmul_pi(a1) : cmul_mi(a1);
        const Cx<R> x0 = a0;
        a2 = csub(x0, a1);
        a0 = cadd(x0, a1);
        a1 = cadd(x0, t);
        a3 = csub(x0, t);
    } else {
        Cx<R> t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3), t3 = csub(a1, a3);
        t3 = INV ? cmul_pi(t3) : cmul_mi(t3);
        a0 = cadd(t0, t2);
        a1 = cadd(t1, t3);
        if constexpr (PART != HALF_OUT) {
            a2 = csub(t0, t2);
            a3 = csub(t1, t3);
        }
    }
}
// e + f q (into x) and e - f q (into y, unless only the first half is wanted)
template <typename R, int PART>
__device__ __forceinline__ void pm_fma(Cx<R>& x, Cx<R>& y, Cx<R> e, Cx<R> q, Kc<R> f) {
    if constexpr (std::is_same<R, Fx>::value) {  // one product for both signs
        const Cx<R> p = cx<R>(fx_mul_const(q.x, f), fx_mul_const(q.y, f));
        x = cadd(e, p);
        if constexpr (PART != HALF_OUT) y = csub(e, p);
        return;
    }
    x.x = fmar(f, q.x, e.x);
    x.y = fmar(f, q.y, e.y);
    if constexpr (PART != HALF_OUT) {
        y.x = fmar(-f, q.x, e.x);
        y.y = fmar(-f, q.y, e.y);
    }
}
template <typename R, int PART>
__device__ __forceinline__ void pm(Cx<R>& x, Cx<R>& y, Cx<R> e, Cx<R> o) {
    x = cadd(e, o);
    if constexpr (PART != HALF_OUT) y = csub(e, o);
}
template <typename R, bool INV, int PART>
__device__ __forceinline__ void dftp8(Cx<R>* v) {
    Cx<R> e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    constexpr int IN = PART == HALF_IN ? HALF_IN : DFT_FULL;
    dftp4<R, INV, IN>(e0, e1, e2, e3);
    dftp4<R, INV, IN>(o0, o1, o2, o3);
    const Kc<R> h = Kc<R>(0.70710678118654752440);
    // w8 = h (1 -+ i), w8^3 = h (-1 -+ i)
    const Cx<R> q1 = INV ? cx<R>(o1.x - o1.y, o1.x + o1.y) : cx<R>(o1.x + o1.y, o1.y - o1.x);
    const Cx<R> q3 = INV ? cx<R>(o3.x + o3.y, o3.y - o3.x) : cx<R>(o3.x - o3.y, o3.x + o3.y);
    pm<R, PART>(v[0], v[4], e0, o0);
    pm_fma<R, PART>(v[1], v[5], e1, q1, h);
    pm<R, PART>(v[2], v[6], e2, INV ? cmul_pi(o2) : cmul_mi(o2));
    pm_fma<R, PART>(v[3], v[7], e3, q3, -h);
}
template <typename R, bool INV, int PART>
__device__ __forceinline__ void dftp16(Cx<R>* v) {
    Cx<R> e[8], o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        e[i] = v[2 * i];
        o[i] = v[2 * i + 1];
    }
    constexpr int IN = PART == HALF_IN ? HALF_IN : DFT_FULL;
    dftp8<R, INV, IN>(e);
    dftp8<R, INV, IN>(o);
    const Kc<R> c = Kc<R>(0.92387953251128675613), t = Kc<R>(0.41421356237309504880), h = Kc<R>(0.70710678118654752440);
    const Kc<R> g = INV ? t : -t;       // w16 = c (1 + i g), w16^7 = -c (1 - i g)
    // w16^3 = c (t + i sg), w16^5 = c (-t + i sg), sg = +-1
    const Cx<R> q1 = cx<R>(fmar(-g, o[1].y, o[1].x), fmar(g, o[1].x, o[1].y));
    const Cx<R> q2 = INV ? cx<R>(o[2].x - o[2].y, o[2].x + o[2].y) : cx<R>(o[2].x + o[2].y, o[2].y - o[2].x);
    const Cx<R> q3 = INV ? cx<R>(fmar(t, o[3].x, -o[3].y), fmar(t, o[3].y, o[3].x))
                           : cx<R>(fmar(t, o[3].x, o[3].y), fmar(t, o[3].y, -o[3].x));
    const Cx<R> q5 = INV ? cx<R>(fmar(-t, o[5].x, -o[5].y), fmar(-t, o[5].y, o[5].x))
                           : cx<R>(fmar(-t, o[5].x, o[5].y), fmar(-t, o[5].y, -o[5].x));
    const Cx<R> q6 = INV ? cx<R>(o[6].x + o[6].y, o[6].y - o[6].x) : cx<R>(o[6].x - o[6].y, o[6].x + o[6].y);
    const Cx<R> q7 = cx<R>(fmar(g, o[7].y, o[7].x), fmar(-g, o[7].x, o[7].y));
    pm<R, PART>(v[0], v[8], e[0], o[0]);
    pm_fma<R, PART>(v[1], v[9], e[1], q1, c);
    pm_fma<R, PART>(v[2], v[10], e[2], q2, h);
    pm_fma<R, PART>(v[3], v[11], e[3], q3, c);
    pm<R, PART>(v[4], v[12], e[4], INV ? cmul_pi(o[4]) : cmul_mi(o[4]));
    pm_fma<R, PART>(v[5], v[13], e[5], q5, c);
    pm_fma<R, PART>(v[6], v[14], e[6], q6, -h);
    pm_fma<R, PART>(v[7], v[15], e[7], q7, -c);
}
// 12 points, n = 4 n1 + n2, k = k1 + 3 k2 (dft12)
template <typename R, bool INV, int PART>
__device__ __forceinline__ void dftp12(Cx<R>* v) {
    Cx<R> y[4][3];
    const Kc<R> s3 = INV ? Kc<R>(-0.86602540378443864676) : Kc<R>(0.86602540378443864676);
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
        const Cx<R> a = v[n2], b = v[4 + n2], c = v[8 + n2];
        if (PART == HALF_IN && n2 >= 2) {  // b = c = 0
            y[n2][0] = y[n2][1] = y[n2][2] = a;
        } else {
            const Cx<R> t = PART == HALF_IN ? b : cadd(b, c), d = PART == HALF_IN ? b : csub(b, c);
            const Cx<R> m = cx<R>(fmar(Kc<R>(-0.5), t.x, a.x), fmar(Kc<R>(-0.5), t.y, a.y));
            y[n2][0] = cadd(a, t);
            y[n2][1] = cx<R>(fmar(s3, d.y, m.x), fmar(-s3, d.x, m.y));
            y[n2][2] = cx<R>(fmar(-s3, d.y, m.x), fmar(s3, d.x, m.y));
        }
    }
    const Kc<R> r3 = Kc<R>(0.86602540378443864676), hf = Kc<R>(0.5);
    const Kc<R> sr3 = INV ? r3 : -r3, shf = INV ? hf : -hf;
    y[1][1] = cmulc<R>(y[1][1], r3, shf);
    y[1][2] = cmulc<R>(y[1][2], hf, sr3);
    y[2][1] = cmulc<R>(y[2][1], hf, sr3);
    y[2][2] = cmulc<R>(y[2][2], -hf, sr3);
    y[3][1] = INV ? cmul_pi(y[3][1]) : cmul_mi(y[3][1]);
    y[3][2] = cx<R>(-y[3][2].x, -y[3][2].y);
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) {
        Cx<R> a0 = y[0][k1], a1 = y[1][k1], a2 = y[2][k1], a3 = y[3][k1];
        dftp4<R, INV, PART == HALF_OUT ? HALF_OUT : DFT_FULL>(a0, a1, a2, a3);
        v[k1] = a0;
        v[k1 + 3] = a1;
        if (PART != HALF_OUT) {
            v[k1 + 6] = a2;
            v[k1 + 9] = a3;
        }
    }
}
template <typename R, bool INV, int P, int PART>
__device__ __forceinline__ void dft_reg(Cx<R>* v) {
    if constexpr (P == 8) dftp8<R, INV, PART>(v);
    else if constexpr (P == 12) dftp12<R, INV, PART>(v);
    else dftp16<R, INV, PART>(v);
}

// v * w (forward) or v * conj(w) (inverse), with fused multiply-adds
template <typename R, bool INV>
__device__ __forceinline__ Cx<R> twmul(Cx<R> v, Cx<R> w) {
    if (INV) return cx<R>(fmar(v.x, w.x, v.y * w.y), fmar(v.y, w.x, -(v.x * w.y)));
    return cx<R>(fmar(v.x, w.x, -(v.y * w.y)), fmar(v.x, w.y, v.y * w.x));
}
template <bool INV>
__device__ __forceinline__ Cx<Fx> twmul(Cx<Fx> v, FxW w) {
    if (INV) return cx<Fx>(fx_mul2(v.x, w.r, v.y, w.i), fx_mul2(v.y, w.r, -v.x, w.i));
    return cx<Fx>(fx_mul2(v.x, w.r, -v.y, w.i), fx_mul2(v.x, w.i, v.y, w.r));
}

// Q of the factorisation L = P * Q of the two-step lengths; 0: the Stockham
// passes
__host__ __device__ constexpr int two_step_q(int L) {
    return L == 64 ? 8 : (L == 96 ? 12 : (L == 128 || L == 192 || L == 256 ? 16 : 0));
}

// The steps of the two-step form in block fixed point (sc_fx.cuh), one work
// item each; tab: the line's table, tw: the twiddles as tw2.  The first steps
// return the magnitude of what they stored: the line's largest decides how far
// the second steps shift the table down to make room for their growth (no bits
// are given up where the line leaves room, and a line's spike costs only
// what it needs).
template <int L>
struct FxSteps {
    static constexpr int Q = two_step_q(L), P = L / Q, ROW = Q + 1;
    static constexpr int B_HALF = fx_bit(P / 2), B_FULL = fx_bit(P), B_INV = fx_bit(Q);  // input bits
    template <bool INV>
    static __device__ __forceinline__ unsigned tw_put(Fx2 v, FxW w, bool one, Fx2* dst) {
        const Fx2 t = one ? v : twmul<INV>(v, w);
        *dst = t;
        return max(fx_mag(t.x), fx_mag(t.y));
    }
    // P-point DFTs first: v[n1] = x[Q n1 + m]
    template <bool INV, int PART>
    static __device__ __forceinline__ unsigned first(Fx2 (&v)[P], int m, const FxW* tw, Fx2* tab) {
        dft_reg<Fx, INV, P, PART>(v);
        unsigned mag = 0;
#pragma unroll
        for (int k1 = 0; k1 < P; ++k1)
            mag = max(mag, tw_put<INV>(v[k1], tw[k1 * Q + m], k1 == 0, tab + k1 * ROW + m));
        return mag;
    }
    // then u[k2] = X[k1 + P k2]
    template <bool INV>
    static __device__ __forceinline__ void second(Fx2 (&u)[Q], int k1, const Fx2* tab, int sh) {
#pragma unroll
        for (int n2 = 0; n2 < Q; ++n2) u[n2] = fx_down(tab[k1 * ROW + n2], sh);
        dft_reg<Fx, INV, Q, DFT_FULL>(u);
    }
    // the transposed flow: Q-point DFTs first, v[n2] = X[n1 + P n2]
    static __device__ __forceinline__ unsigned t_first(Fx2 (&v)[Q], int n1, const FxW* tw, Fx2* tab) {
        dft_reg<Fx, true, Q, DFT_FULL>(v);
        unsigned mag = 0;
#pragma unroll
        for (int k2 = 0; k2 < Q; ++k2)
            mag = max(mag, tw_put<true>(v[k2], tw[n1 * Q + k2], k2 == 0, tab + n1 * ROW + k2));
        return mag;
    }
    // then u[k1] = x[Q k1 + k2], k1 < P / 2
    static __device__ __forceinline__ void t_second(Fx2 (&u)[P], int k2, const Fx2* tab, int sh) {
#pragma unroll
        for (int n1 = 0; n1 < P; ++n1) u[n1] = fx_down(tab[n1 * ROW + k2], sh);
        dft_reg<Fx, true, P, HALF_OUT>(u);
    }
};

}  // namespace ocsc
