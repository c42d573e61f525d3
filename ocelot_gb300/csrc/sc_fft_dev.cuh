// Batched FFTs of lines held in shared memory: mixed-radix (3/2/4/8)
// Stockham passes, and for the common lengths (64 to 256) the two-step form below.
//
// The lines of one thread block live in shared memory, line l at a + l*ls,
// elements contiguous.  Each stage reads radix-r butterfly inputs with stride
// L/r, applies the twiddles w^(t*k), does the r-point DFT in registers and
// writes the outputs in autosorted (Stockham) order into the other buffer, so
// no bit reversal is needed.  Twiddles come from a per-block table in
// shared memory built from tw[m] = exp(-2*pi*i*m/L) (load_twiddles: one block
// of entries per stage, read by consecutive lanes); the inverse uses their
// conjugates and leaves the 1/L normalisation to the caller.
#pragma once
#include "sc_common.cuh"
#include "sc_dft.cuh"

namespace ocsc {

template <typename C, bool INV>
__device__ __forceinline__ void dft2(C& a, C& b) {
    C t = a;
    a = cadd(t, b);
    b = csub(t, b);
}

template <typename C, bool INV>
__device__ __forceinline__ void dft4(C& a0, C& a1, C& a2, C& a3) {
    C t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3), t3 = csub(a1, a3);
    t3 = INV ? cmul_pi(t3) : cmul_mi(t3);
    a0 = cadd(t0, t2);
    a2 = csub(t0, t2);
    a1 = cadd(t1, t3);
    a3 = csub(t1, t3);
}

// 3-point DFT: y_k = sum_t a_t w^(t k), w = exp(-2 pi i / 3) (forward) or its
// conjugate (inverse): y0 = a + (b + c), y1,2 = a - (b + c)/2 -/+ i (sqrt(3)/2)(b - c)
template <typename R, bool INV>
__device__ __forceinline__ void dft3(Cx<R>& a, Cx<R>& b, Cx<R>& c) {
    const R s = INV ? (R)-0.86602540378443864676 : (R)0.86602540378443864676;
    const Cx<R> t = cadd(b, c), d = csub(b, c);
    const Cx<R> m = cx<R>(a.x - (R)0.5 * t.x, a.y - (R)0.5 * t.y);
    const Cx<R> r = cx<R>(s * d.y, -s * d.x);  // -i s d
    a = cadd(a, t);
    b = cadd(m, r);
    c = csub(m, r);
}

template <typename R, bool INV>
__device__ __forceinline__ void dft8(Cx<R>* v) {
    Cx<R> e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    Cx<R> o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    dft4<Cx<R>, INV>(e0, e1, e2, e3);
    dft4<Cx<R>, INV>(o0, o1, o2, o3);
    const R h = (R)0.70710678118654752440;
    if (!INV) {  // w = exp(-i*pi/4)
        o1 = cx<R>((o1.x + o1.y) * h, (o1.y - o1.x) * h);
        o2 = cmul_mi(o2);
        o3 = cx<R>((o3.y - o3.x) * h, (-o3.x - o3.y) * h);
    } else {     // w = exp(+i*pi/4)
        o1 = cx<R>((o1.x - o1.y) * h, (o1.x + o1.y) * h);
        o2 = cmul_pi(o2);
        o3 = cx<R>((-o3.x - o3.y) * h, (o3.x - o3.y) * h);
    }
    v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
    v[1] = cadd(e1, o1); v[5] = csub(e1, o1);
    v[2] = cadd(e2, o2); v[6] = csub(e2, o2);
    v[3] = cadd(e3, o3); v[7] = csub(e3, o3);
}

// tw: the stage twiddle table of load_twiddles; the stage's block starts at
// Ns - (the first stage's radix)
template <typename R, bool INV, int RAD>
__device__ __forceinline__ void stockham_stage(const Cx<R>* __restrict__ a, Cx<R>* __restrict__ b,
                                               int L, int ls, int nl, int Ns, const Cx<R>* tw, int tw_off) {
    const int nb = L / RAD;
    const int total = nb * nl;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int line = idx / nb;
        const int j = idx - line * nb;
        const Cx<R>* src = a + line * ls;
        Cx<R>* dst = b + line * ls;
        const int k = j % Ns;
        Cx<R> v[RAD];
#pragma unroll
        for (int t = 0; t < RAD; ++t) v[t] = src[j + t * nb];
        if (Ns > 1) {
#pragma unroll
            for (int t = 1; t < RAD; ++t) {
                Cx<R> w = tw[tw_off + (t - 1) * Ns + k];
                if (INV) w.y = -w.y;
                v[t] = cmul(v[t], w);
            }
        }
        if (RAD == 2) dft2<Cx<R>, INV>(v[0], v[1]);
        else if (RAD == 3) dft3<R, INV>(v[0], v[1], v[2]);
        else if (RAD == 4) dft4<Cx<R>, INV>(v[0], v[1], v[2], v[3]);
        else dft8<R, INV>(v);
        const int out = (j - k) * RAD + k;
#pragma unroll
        for (int t = 0; t < RAD; ++t) dst[out + t * Ns] = v[t];
    }
}

// The same stages with the line length known at compile time: the radix of
// each stage, the butterfly count and the twiddle stride are constants, so
// the index arithmetic reduces to shifts, masks and multiplications.  The
// plan is the one of make_radix_plan (for lengths 3 * 2^k one radix-3 stage,
// then radix 8 while it divides, then 4, then 2) and the arithmetic is that
// of stockham_stage, so results are identical.
constexpr int plan_radix(int L, int s) {
    int rem = L, st = 0;
    if (rem % 3 == 0) {
        if (st == s) return 3;
        rem /= 3;
        ++st;
    }
    while (rem % 8 == 0 && rem > 1) {
        if (st == s) return 8;
        rem /= 8;
        ++st;
    }
    while (rem % 4 == 0 && rem > 1) {
        if (st == s) return 4;
        rem /= 4;
        ++st;
    }
    while (rem % 2 == 0 && rem > 1) {
        if (st == s) return 2;
        rem /= 2;
        ++st;
    }
    return 0;
}

// Intermediate stages keep element i of a line at a padded position: the
// Stockham output index of the early stages strides by RAD elements per
// thread, which in the plain layout puts 8 or more threads of a warp on the
// same bank.  One pad element per 16 (lines of 128 points and more) spreads
// those strides over all banks and keeps the 16 lanes of a half-warp that
// read consecutive elements on 16 distinct bank pairs; with one pad per 8 the
// half-warp's 16 elements spanned 17 slots and its first and last lane met on
// one bank (a shared-memory model of the stages: 11% fewer wavefronts at 128
// points, 10% at 512).  Shorter lines keep one pad per 8, which is as good or
// better there.  The first stage reads and the last one writes the plain
// layout the kernels load and store; the padded line fits in fft_ls(L).
template <int L>
__device__ __forceinline__ int fft_pad(int i) {
    return L >= 128 ? i + (i >> 4) : i + (i >> 3);
}

// tw: the stage twiddle table of load_twiddles (this stage's block at
// NS - plan_radix(L, 0), entry (t - 1) NS + k = w_L^(t k L / (NS RAD)))
template <typename R, bool INV, int RAD, int L, int NS, bool PIN, bool POUT>
__device__ __forceinline__ void stockham_stage_c(const Cx<R>* __restrict__ a, Cx<R>* __restrict__ b, int ls,
                                                 int nl, const Cx<R>* tw) {
    constexpr int nb = L / RAD;
    constexpr int tw_off = NS - plan_radix(L, 0);
    const int total = nb * nl;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int line = idx / nb;
        const int j = idx - line * nb;
        const int k = j % NS;
        const Cx<R>* src = a + line * ls;
        Cx<R>* dst = b + line * ls;
        Cx<R> v[RAD];
#pragma unroll
        for (int t = 0; t < RAD; ++t) v[t] = src[PIN ? fft_pad<L>(j + t * nb) : j + t * nb];
        if (NS > 1) {
#pragma unroll
            for (int t = 1; t < RAD; ++t) {
                Cx<R> w = tw[tw_off + (t - 1) * NS + k];
                if (INV) w.y = -w.y;
                v[t] = cmul(v[t], w);
            }
        }
        if (RAD == 2) dft2<Cx<R>, INV>(v[0], v[1]);
        else if (RAD == 3) dft3<R, INV>(v[0], v[1], v[2]);
        else if (RAD == 4) dft4<Cx<R>, INV>(v[0], v[1], v[2], v[3]);
        else dft8<R, INV>(v);
        const int out = (j - k) * RAD + k;
#pragma unroll
        for (int t = 0; t < RAD; ++t) dst[POUT ? fft_pad<L>(out + t * NS) : out + t * NS] = v[t];
    }
}

// ---------------------------------------------------------------------------
// Two-step FFT (sc_dft.cuh) of lines in shared memory
// ---------------------------------------------------------------------------
// ls >= fft_ls(L) >= P (Q + 1); a holds the input, b is scratch; the result is
// returned in a.  LF: nl is a power of two, lg its log2.  Called by every thread
// of the block; ends with a barrier.  HALF: the passes of the
// zero-padded convolution, whose forward lines are zero past the mesh (at most
// L / 2 points) and whose inverse lines are only read up to it.  Forward (and
// without HALF): the P-point DFTs first, over inputs of which
// the second half is zero.  Inverse with HALF: the transposed flow
//   x[Q k1 + k2] = sum_n1 w_P^(n1 k1) w_L^(n1 k2) sum_n2 w_Q^(n2 k2) X[n1 + P n2],
// the Q-point DFTs first, then P-point ones of which the first half of the
// outputs is kept; the twiddles are the same table w_L^(n1 k2) at n1 * Q + k2.
// One shared-memory round trip per step.  FP32 lines; double ones go through fft_fx.
template <typename R, bool INV, int L, bool LF, bool HALF>
__device__ __forceinline__ Cx<R>* fft_two_step(Cx<R>* a, Cx<R>* b, int ls, int nl, int lg, const Cx<R>* tw2) {
    constexpr int Q = two_step_q(L), P = L / Q;
    static_assert(Q > 0 && P * Q == L && P <= Q && P * (Q + 1) <= fft_ls(L), "two-step factorisation");
    constexpr bool T = INV && HALF;             // the transposed flow
    constexpr int A = T ? P : Q, B = T ? Q : P;  // work items per line of the first and of the second step
    auto split = [&](int idx, int per, int& line, int& m) {
        if (LF) {
            m = idx >> lg;
            line = idx & (nl - 1);
        } else {
            line = idx / per;
            m = idx - line * per;
        }
    };
    for (int idx = threadIdx.x; idx < nl * A; idx += blockDim.x) {
        int line, m;
        split(idx, A, line, m);
        const Cx<R>* src = a + line * ls + m;
        if constexpr (T) {
            Cx<R> v[Q];
#pragma unroll
            for (int n2 = 0; n2 < Q; ++n2) v[n2] = src[n2 * P];
            dft_reg<R, INV, Q, DFT_FULL>(v);
            Cx<R>* dst = b + line * ls + m * (Q + 1);
            dst[0] = v[0];
#pragma unroll
            for (int k2 = 1; k2 < Q; ++k2) dst[k2] = twmul<R, INV>(v[k2], tw2[m * Q + k2]);
        } else {
            Cx<R> v[P];
#pragma unroll
            for (int n1 = 0; n1 < P; ++n1)
                if (!HALF || n1 < P / 2) v[n1] = src[n1 * Q];
            dft_reg<R, INV, P, HALF ? HALF_IN : DFT_FULL>(v);
            Cx<R>* dst = b + line * ls + m;
            dst[0] = v[0];
#pragma unroll
            for (int k1 = 1; k1 < P; ++k1) dst[k1 * (Q + 1)] = twmul<R, INV>(v[k1], tw2[k1 * Q + m]);
        }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < nl * B; idx += blockDim.x) {
        int line, m;
        split(idx, B, line, m);
        if constexpr (T) {
            const Cx<R>* src = b + line * ls + m;
            Cx<R> u[P];
#pragma unroll
            for (int n1 = 0; n1 < P; ++n1) u[n1] = src[n1 * (Q + 1)];
            dft_reg<R, INV, P, HALF_OUT>(u);
            Cx<R>* dst = a + line * ls + m;
#pragma unroll
            for (int k1 = 0; k1 < P / 2; ++k1) dst[k1 * Q] = u[k1];
        } else {
            const Cx<R>* src = b + line * ls + m * (Q + 1);
            Cx<R> u[Q];
#pragma unroll
            for (int n2 = 0; n2 < Q; ++n2) u[n2] = src[n2];
            dft_reg<R, INV, Q, DFT_FULL>(u);
            Cx<R>* dst = a + line * ls + m;
#pragma unroll
            for (int k2 = 0; k2 < Q; ++k2) dst[k2 * P] = u[k2];
        }
    }
    __syncthreads();
    return a;
}

// fft_two_step for double lines (lg >= 0: line-fastest).  Each line's exponent and
// table magnitude stand in the slot after its table.
template <bool INV, int L, bool HALF>
__device__ __forceinline__ Cx<double>* fft_fx(Cx<double>* a, Cx<double>* b, int ls, int nl, int lg,
                                              const Cx<double>* tw2) {
    using S = FxSteps<L>;
    constexpr int Q = S::Q, P = S::P, SLOT = P * S::ROW;
    static_assert(Q > 0 && P * Q == L && P <= Q && SLOT < fft_ls(L), "two-step factorisation");
    constexpr bool T = INV && HALF;             // the transposed flow
    constexpr int A = T ? P : Q, B = T ? Q : P;  // work items per line of the first and of the second step
    constexpr int NIN = T ? Q : (HALF ? P / 2 : P);  // inputs of an item of the first step
    constexpr int BIT = T ? S::B_INV : (HALF ? S::B_HALF : S::B_FULL);
    const FxW* tw = reinterpret_cast<const FxW*>(tw2);
    Fx2* tb = reinterpret_cast<Fx2*>(b);
    auto slot = [&](int line) { return reinterpret_cast<int*>(tb + line * ls + SLOT); };
    auto split = [&](int idx, int per, int& line, int& m) {
        if (lg >= 0) {
            m = idx >> lg;
            line = idx & (nl - 1);
        } else {
            line = idx / per;
            m = idx - line * per;
        }
    };
    for (int l = threadIdx.x; l < nl; l += blockDim.x) {
        slot(l)[0] = 1;  // the exponent of denormals
        slot(l)[1] = 0;
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < nl * A; idx += blockDim.x) {
        int line, m, e = 0;
        split(idx, A, line, m);
#pragma unroll
        for (int n = 0; n < NIN; ++n) {
            const Cx<double> c = a[line * ls + m + n * A];
            e = max(e, max(fx_exp(c.x), fx_exp(c.y)));
        }
        atomicMax(slot(line), e);
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < nl * A; idx += blockDim.x) {
        int line, m;
        split(idx, A, line, m);
        const int E = slot(line)[0];
        Fx2 v[T ? Q : P];
#pragma unroll
        for (int n = 0; n < NIN; ++n) {
            const Cx<double> c = a[line * ls + m + n * A];
            v[n] = cx<Fx>(fx_from<BIT>(c.x, E), fx_from<BIT>(c.y, E));
        }
        unsigned mag;
        if constexpr (T) mag = S::t_first(v, m, tw, tb + line * ls);
        else mag = S::template first<INV, HALF ? HALF_IN : DFT_FULL>(v, m, tw, tb + line * ls);
        atomicMax(slot(line) + 1, (int)mag);
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < nl * B; idx += blockDim.x) {
        int line, m;
        split(idx, B, line, m);
        const int* sl = slot(line);
        const int sh = fx_room<T ? P : Q>((unsigned)sl[1]);
        const FxOut o(sl[0], BIT - sh);
        Fx2 u[T ? P : Q];
        if constexpr (T) S::t_second(u, m, tb + line * ls, sh);
        else S::template second<INV>(u, m, tb + line * ls, sh);
        Cx<double>* dst = a + line * ls + m;
#pragma unroll
        for (int k = 0; k < (T ? P / 2 : Q); ++k) dst[k * B] = cx<double>(fx_to(u[k].x, o), fx_to(u[k].y, o));
    }
    __syncthreads();
    return a;
}
template <typename R, bool INV, int L, bool HALF>
__device__ __forceinline__ Cx<R>* fft_two_step_any(Cx<R>* a, Cx<R>* b, int ls, int nl, const Cx<R>* tw2) {
    if constexpr (sizeof(R) == 8) {
        return fft_fx<INV, L, HALF>(a, b, ls, nl, nl >= 8 && (nl & (nl - 1)) == 0 ? 31 - __clz(nl) : -1, tw2);
    } else {
        if (nl >= 16 && (nl & (nl - 1)) == 0)
            return fft_two_step<R, INV, L, true, HALF>(a, b, ls, nl, 31 - __clz(nl), tw2);
        return fft_two_step<R, INV, L, false, HALF>(a, b, ls, nl, 0, tw2);
    }
}

// ls must be at least fft_ls(L)
template <typename R, bool INV, int L, int S, int NS>
__device__ __forceinline__ Cx<R>* fft_stages_c(Cx<R>* a, Cx<R>* b, int ls, int nl, const Cx<R>* tw) {
    constexpr int RAD = plan_radix(L, S);
    if constexpr (RAD == 0) {
        return a;
    } else {
        stockham_stage_c<R, INV, RAD, L, NS, (S > 0), (plan_radix(L, S + 1) != 0)>(a, b, ls, nl, tw);
        __syncthreads();
        return fft_stages_c<R, INV, L, S + 1, NS * RAD>(b, a, ls, nl, tw);
    }
}

// Whether a line length takes the two-step form (its twiddle table then stays
// w_L^m in the workspace, the stage table otherwise).
__host__ __device__ constexpr bool uses_two_step(int L) { return two_step_q(L) != 0; }

template <int V>
struct IntC {
    static constexpr int value = V;
};
// f(IntC<L>) on the host for a two-step length L
template <typename F>
static cudaError_t two_step_host(int L, F&& f) {
    switch (L) {
        case 64: return f(IntC<64>{});
        case 96: return f(IntC<96>{});
        case 128: return f(IntC<128>{});
        case 192: return f(IntC<192>{});
        case 256: return f(IntC<256>{});
        default: return cudaErrorInvalidValue;
    }
}
static_assert(uses_two_step(64) && uses_two_step(96) && uses_two_step(128) && uses_two_step(192) &&
                  uses_two_step(256) && !uses_two_step(32) && !uses_two_step(48) && !uses_two_step(384) &&
                  !uses_two_step(512),
              "two_step_host lists the two-step lengths");

// FFT of nl lines of length rp.L; a holds the input, b is scratch of the
// same shape.  Returns the buffer that holds the result.  Must be called by
// every thread of the block; ends with a barrier.  HALF (the convolution's
// passes): the caller's input is zero from L / 2 on (forward) or it reads only
// the first L / 2 results (inverse; the rest may not be written).
// TWO: false where the caller has other code for the two-step lengths.
template <typename R, bool INV, bool HALF = false, bool TWO = true>
__device__ Cx<R>* fft_lines(Cx<R>* a, Cx<R>* b, int ls, int nl, const RadixPlan& rp, const Cx<R>* tw) {
    if constexpr (TWO) {
        switch (rp.L) {
            case 64: return fft_two_step_any<R, INV, 64, HALF>(a, b, ls, nl, tw);
            case 96: return fft_two_step_any<R, INV, 96, HALF>(a, b, ls, nl, tw);
            case 128: return fft_two_step_any<R, INV, 128, HALF>(a, b, ls, nl, tw);
            case 192: return fft_two_step_any<R, INV, 192, HALF>(a, b, ls, nl, tw);
            case 256: return fft_two_step_any<R, INV, 256, HALF>(a, b, ls, nl, tw);
            default: break;
        }
    }
    switch (rp.L) {  // the padded lengths of meshes up to 256 per axis
        case 8: return fft_stages_c<R, INV, 8, 0, 1>(a, b, ls, nl, tw);
        case 12: return fft_stages_c<R, INV, 12, 0, 1>(a, b, ls, nl, tw);
        case 16: return fft_stages_c<R, INV, 16, 0, 1>(a, b, ls, nl, tw);
        case 24: return fft_stages_c<R, INV, 24, 0, 1>(a, b, ls, nl, tw);
        case 32: return fft_stages_c<R, INV, 32, 0, 1>(a, b, ls, nl, tw);
        case 48: return fft_stages_c<R, INV, 48, 0, 1>(a, b, ls, nl, tw);
        case 384: return fft_stages_c<R, INV, 384, 0, 1>(a, b, ls, nl, tw);
        case 512: return fft_stages_c<R, INV, 512, 0, 1>(a, b, ls, nl, tw);
        default: break;
    }
    int Ns = 1;
    for (int s = 0; s < rp.nst; ++s) {
        const int r = rp.r[s], off = Ns - rp.r[0];
        if (r == 8) stockham_stage<R, INV, 8>(a, b, rp.L, ls, nl, Ns, tw, off);
        else if (r == 4) stockham_stage<R, INV, 4>(a, b, rp.L, ls, nl, Ns, tw, off);
        else if (r == 3) stockham_stage<R, INV, 3>(a, b, rp.L, ls, nl, Ns, tw, off);
        else stockham_stage<R, INV, 2>(a, b, rp.L, ls, nl, Ns, tw, off);
        __syncthreads();
        Cx<R>* t = a;
        a = b;
        b = t;
        Ns *= r;
    }
    return a;
}

// the radix of the next Stockham stage of a line with rem points left to
// split (the order of plan_radix / make_radix_plan: a 3 first, then 8s, a 4,
// a 2)
__host__ __device__ inline int next_radix(int rem) {
    return rem % 3 == 0 ? 3 : (rem % 8 == 0 ? 8 : (rem % 4 == 0 ? 4 : 2));
}

// The Stockham stage twiddle table: one block per stage after the first, in
// stage order -- the stage of NS points per butterfly group and radix RAD
// holds w_L^(t k L / (NS RAD)) at (t - 1) NS + k for t = 1 .. RAD - 1, k < NS,
// and starts at NS - R0 (R0 the first radix; L - R0 entries in all) -- so that
// lanes with consecutive k read consecutive entries (read from a table of
// w_L^m by m = t k L / (NS RAD), the 512-point stages put up to 8 lanes on one
// bank).  stage_tw_exponent gives the m of entry i < L - R0; the workspace's
// twiddle tables are laid out this way once, when it is initialised.
__host__ __device__ inline int stage_tw_exponent(int L, int i) {
    const int r0 = next_radix(L);
    const int g = i + r0;   // the stage of entry i: NS <= g < NS * RAD
    int ns = r0, rem = L / r0, r = next_radix(rem);
    while (ns * r <= g) {
        ns *= r;
        rem /= r;
        r = next_radix(rem);
    }
    const int rel = g - ns, t = rel / ns + 1, k = rel - (t - 1) * ns;
    return t * k * (L / (ns * r));
}

// The twiddle table of fft_lines in shared memory (room for L entries) from
// the workspace's table src: for the two-step lengths src[m] = w_L^m
// and tw2[k1 * Q + n2] = w_L^(n2 k1) is formed here; for the Stockham lengths
// src already holds the stage table and is copied.
template <typename R>
__device__ __forceinline__ void load_twiddles(Cx<R>* dst, const Cx<R>* src, int L) {
    const int Q = two_step_q(L);
    if (Q) {
        for (int i = threadIdx.x; i < L; i += blockDim.x) {
            const int k1 = i / Q, n2 = i - k1 * Q;
            dst[i] = src[k1 * n2];
        }
        return;
    }
    for (int i = threadIdx.x; i < L; i += blockDim.x) dst[i] = src[i];
}

// Quotient and remainder of i = start, start + step, start + 2 step, ... by d,
// carried from one to the next: two divisions per thread instead of one per
// element in the line-staging loops (d is a run-time line length).
struct DivWalk {
    int q, r, dq, dr, d;
    __device__ __forceinline__ DivWalk(int start, int step, int d_) : d(d_) {
        q = start / d;
        r = start - q * d;
        dq = step / d;
        dr = step - dq * d;
    }
    __device__ __forceinline__ void next() {
        q += dq;
        r += dr;
        if (r >= d) {
            r -= d;
            ++q;
        }
    }
};

// Columns of a strided pass: the block's TK columns (TK a power of two) are
// consecutive entries of a flattened column index, thread t takes column
// t mod TK and rows t / TK, t / TK + blockDim / TK, ...; no division per element.
struct ColMap {
    int kk, r0, rs;
    __device__ __forceinline__ explicit ColMap(int TK) {
        const int lg = 31 - __clz(TK);
        kk = threadIdx.x & (TK - 1);
        r0 = threadIdx.x >> lg;
        rs = blockDim.x >> lg;
    }
};

}  // namespace ocsc
