// The FP32 convolution's column passes and z forward pass for line lengths of
// the two-step form, with the lines streamed: each step's register DFTs take
// their inputs straight from global memory and give their outputs straight to
// it, so a transform costs one shared-memory round trip (the table between its
// two steps) and one barrier.
// The passes that stage whole lines first (sc_fft.cu, other lengths) write and
// read shared memory three times more per transform, with a barrier each.  The
// DFTs, twiddles and products are those of fft_two_step, in the same order, so
// the plane-fused passes give the same bits.
//
// What bounds them on GB300: at 64^3 (one wave of blocks) the latency of the
// global loads and of the two steps; at 128 x 128 x 256 and in batches the
// issue rate and the L2/HBM round trips.  Measured, Stockham or staged two-step
// -> streamed: 32^3 x pass 6.6 -> 3.9 us; 64^3 x pass 14.9 -> 8.1, y inverse 9.9 ->
// 5.9, z forward 6.3 -> 6.0; 128 x 128 x 256 x pass 148 -> 97, y 33/106 -> 20/88; 16 uneven beams
// x 125 -> 76, y 31/87 -> 23/60.  Not streamed, because measured slower so: the z
// inverse (its step reads strided entries of two rows; 8.8 -> 9.6 us at 64^3).
// The FP64 form's passes are in sc_fft_fx.cuh.
#pragma once
#include "sc_fft_dev.cuh"

namespace ocsc {

// whether lines of length L are streamed
template <typename R>
__host__ __device__ constexpr bool streamed(int L) { return sizeof(R) == 4 && uses_two_step(L); }

// f(IntC<L>) for a streamed length L; false (and nothing done) for any other
template <typename R, typename F>
__device__ __forceinline__ bool with_stream(int L, F&& f) {
    if constexpr (sizeof(R) == 4) {
        switch (L) {
            case 64: f(IntC<64>{}); return true;
            case 96: f(IntC<96>{}); return true;
            case 128: f(IntC<128>{}); return true;
            case 192: f(IntC<192>{}); return true;
            case 256: f(IntC<256>{}); return true;
            default: break;
        }
    }
    return false;
}
static_assert(streamed<float>(64) && streamed<float>(96) && streamed<float>(128) && streamed<float>(192) &&
                  streamed<float>(256) && !streamed<float>(32) && !streamed<float>(512),
              "with_stream lists the streamed lengths");

// threads of a streamed column pass over 16 columns: an item each in the wider step
constexpr int stream_threads(int L) { return 16 * two_step_q(L); }
// blocks per SM they are compiled for: 64 registers (without the bound the
// 128-point x pass takes 74, and the batched passes 97 us instead of 85)
constexpr int stream_minb(int L) { return 1024 / stream_threads(L); }

// strides of a line's table between the steps and of a line in natural order
template <typename R>
__host__ __device__ constexpr int stream_lb(int L) {
    return streamed<R>(L) ? ((L / two_step_q(L)) * (two_step_q(L) + 1)) | 1 : 0;
}
__host__ __device__ constexpr int stream_la(int L) { return L | 1; }
// whether the x pass holds the tables of both its inverse transforms at once
// (then they share their barriers and fill the block; 52 KB at 128 points, four
// blocks per SM; 104 KB at 256 would leave two)
__host__ __device__ constexpr bool stream_dual_x(int L) { return L <= 128; }

// the four register steps; dst / src: the line's table (+ the item's offset)
template <typename R, int L>
struct Steps {
    static constexpr int Q = two_step_q(L), P = L / Q;
    // forward, first: v[0 .. P/2) = x[Q n1 + m] (the rest is zero)
    static __device__ __forceinline__ void fwd1(Cx<R> (&v)[P], int m, const Cx<R>* tw, Cx<R>* tab) {
        dft_reg<R, false, P, HALF_IN>(v);
        tab[m] = v[0];
#pragma unroll
        for (int k1 = 1; k1 < P; ++k1) tab[k1 * (Q + 1) + m] = twmul<R, false>(v[k1], tw[k1 * Q + m]);
    }
    // forward, second: u[k2] = X[k1 + P k2]
    static __device__ __forceinline__ void fwd2(Cx<R> (&u)[Q], int k1, const Cx<R>* tab) {
#pragma unroll
        for (int n2 = 0; n2 < Q; ++n2) u[n2] = tab[k1 * (Q + 1) + n2];
        dft_reg<R, false, Q, DFT_FULL>(u);
    }
    // inverse (transposed flow), first: v[n2] = X[n1 + P n2]
    static __device__ __forceinline__ void inv1(Cx<R> (&v)[Q], int n1, const Cx<R>* tw, Cx<R>* tab) {
        dft_reg<R, true, Q, DFT_FULL>(v);
        Cx<R>* dst = tab + n1 * (Q + 1);
        dst[0] = v[0];
#pragma unroll
        for (int k2 = 1; k2 < Q; ++k2) dst[k2] = twmul<R, true>(v[k2], tw[n1 * Q + k2]);
    }
    // inverse, second: u[k1] = x[Q k1 + k2], k1 < P / 2
    static __device__ __forceinline__ void inv2(Cx<R> (&u)[P], int k2, const Cx<R>* tab) {
#pragma unroll
        for (int n1 = 0; n1 < P; ++n1) u[n1] = tab[n1 * (Q + 1) + k2];
        dft_reg<R, true, P, HALF_OUT>(u);
    }
};

template <typename R>
__device__ __forceinline__ Cx<R> cmul_plain(Cx<R> a, Cx<R> b) {
    return cx<R>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// Column passes: a block's TK columns (a power of two), thread t works on
// column t mod TK, its items t / TK, t / TK + blockDim / TK, ...
//
// y pass, in place on W (as ypass_body).  Forward: rows < ny in, all My out;
// inverse: all in, rows < ny out, and with W3 the columns times D(ky) into W3
// beside them (the second half of the items reads W again).
template <typename R, bool INV, int L>
__device__ __forceinline__ void ypass_stream(Cx<R>* __restrict__ W, int nx, int ny, int Kz,
                                             const Cx<R>* __restrict__ twg, int TK, VBlk vb, Cx<R>* __restrict__ W3,
                                             const Cx<R>* __restrict__ dy) {
    using S = Steps<R, L>;
    constexpr int Q = S::Q, P = S::P, lb = stream_lb<R>(L);
    extern __shared__ __align__(16) unsigned char smraw[];
    Cx<R>* tw = reinterpret_cast<Cx<R>*>(smraw);
    Cx<R>* ds = tw + L;
    Cx<R>* B = ds + (W3 ? L : 0);
    const ColMap cm(TK);
    const int col = vb.x * TK + cm.kk;
    const bool live = col < nx * Kz;
    const int x = col / Kz, k = col - x * Kz;
    const size_t base = (size_t)x * L * Kz + k;  // element y of the column at base + y * Kz
    const int nd = W3 ? 2 : 1;
    auto tab = [&](int t) { return B + (t * TK + cm.kk) * lb; };
    if constexpr (!INV) {
        Cx<R> v[P];
        auto ld = [&](int m) {
#pragma unroll
            for (int n1 = 0; n1 < P / 2; ++n1) {
                const int y = n1 * Q + m;
                v[n1] = (y < ny && live) ? W[base + (size_t)y * Kz] : cx<R>(0, 0);
            }
        };
        if (cm.r0 < Q) ld(cm.r0);
        load_twiddles<R>(tw, twg, L);
        __syncthreads();
        for (int m = cm.r0; m < Q; m += cm.rs) {
            if (m != cm.r0) ld(m);
            S::fwd1(v, m, tw, tab(0));
        }
        __syncthreads();
        for (int k1 = cm.r0; k1 < P; k1 += cm.rs) {
            Cx<R> u[Q];
            S::fwd2(u, k1, tab(0));
            if (live)
#pragma unroll
                for (int k2 = 0; k2 < Q; ++k2) W[base + (size_t)(k1 + P * k2) * Kz] = u[k2];
        }
    } else {
        Cx<R> v[Q];
        auto item = [&](int i, int per, int& which, int& m) {
            which = i >= per;
            m = i - which * per;
        };
        auto ldi = [&](int m) {
#pragma unroll
            for (int n2 = 0; n2 < Q; ++n2) v[n2] = live ? W[base + (size_t)(m + P * n2) * Kz] : cx<R>(0, 0);
        };
        int which, m;
        item(cm.r0, P, which, m);
        if (cm.r0 < nd * P) ldi(m);
        load_twiddles<R>(tw, twg, L);
        if (W3)
            for (int i = threadIdx.x; i < L; i += blockDim.x) ds[i] = dy[i];
        __syncthreads();
        for (int i = cm.r0; i < nd * P; i += cm.rs) {
            item(i, P, which, m);
            if (i != cm.r0) ldi(m);
            if (which)
#pragma unroll
                for (int n2 = 0; n2 < Q; ++n2) v[n2] = cmul_plain<R>(v[n2], ds[m + P * n2]);
            S::inv1(v, m, tw, tab(which));
        }
        __syncthreads();
        for (int i = cm.r0; i < nd * Q; i += cm.rs) {
            item(i, Q, which, m);
            Cx<R> u[P];
            S::inv2(u, m, tab(which));
            Cx<R>* out = which ? W3 : W;
#pragma unroll
            for (int k1 = 0; k1 < P / 2; ++k1) {
                const int y = k1 * Q + m;
                if (live && y < ny) out[base + (size_t)y * Kz] = u[k1];
            }
        }
    }
}

// x pass (as xconv_body): forward over the nx planes, Green multiply, inverse,
// and with W2 the product times D(kx) through its own inverse into W2
template <typename R, int L>
__device__ __forceinline__ void xconv_stream(Cx<R>* __restrict__ W, const R* __restrict__ G, int nx, int My, int Kz,
                                             int Ky, const Cx<R>* __restrict__ twg, int TK, const ScState* st, VBlk vb,
                                             Cx<R>* __restrict__ W2, const Cx<R>* __restrict__ dx) {
    using S = Steps<R, L>;
    constexpr int Q = S::Q, P = S::P, la = stream_la(L), lb = stream_lb<R>(L);
    extern __shared__ __align__(16) unsigned char smraw[];
    Cx<R>* tw = reinterpret_cast<Cx<R>*>(smraw);
    Cx<R>* ds = tw + L;
    Cx<R>* A = ds + (W2 ? L : 0);
    Cx<R>* B = A + TK * la;
    const ColMap cm(TK);
    const int col = vb.x * TK + cm.kk;
    const int ncol = My * Kz;
    const bool live = col < ncol;
    const int ky = col / Kz, k = col - ky * Kz;
    const int gy = ky <= My - ky ? ky : My - ky;
    const int gk = gy * Kz + k;  // the column's Green entry at gx * Ky * Kz + gk
    const int KyKz = Ky * Kz;
    Cx<R>* line = A + cm.kk * la;
    auto tab = [&](int t) { return B + (t * TK + cm.kk) * lb; };
    {
        Cx<R> v[P];
        auto ld = [&](int m) {
#pragma unroll
            for (int n1 = 0; n1 < P / 2; ++n1) {
                const int x = n1 * Q + m;
                v[n1] = (x < nx && live) ? W[(size_t)x * ncol + col] : cx<R>(0, 0);
            }
        };
        if (cm.r0 < Q) ld(cm.r0);
        load_twiddles<R>(tw, twg, L);
        if (W2)
            for (int i = threadIdx.x; i < L; i += blockDim.x) ds[i] = dx[i];
        __syncthreads();
        for (int m = cm.r0; m < Q; m += cm.rs) {
            if (m != cm.r0) ld(m);
            S::fwd1(v, m, tw, tab(0));
        }
    }
    {
        R g[Q];
        auto ldg = [&](int k1) {
#pragma unroll
            for (int k2 = 0; k2 < Q; ++k2) {
                const int kx = k1 + P * k2, gx = kx <= L - kx ? kx : L - kx;
                const long long gi = (long long)gx * KyKz + gk;
                g[k2] = (live && SC_IDX_OK(st, 23, gi, (long long)(L / 2 + 1) * KyKz)) ? G[gi] : (R)0;
            }
        };
        if (cm.r0 < P) ldg(cm.r0);
        __syncthreads();
        for (int k1 = cm.r0; k1 < P; k1 += cm.rs) {
            if (k1 != cm.r0) ldg(k1);
            Cx<R> u[Q];
            S::fwd2(u, k1, tab(0));
#pragma unroll
            for (int k2 = 0; k2 < Q; ++k2) line[k1 + P * k2] = cx<R>(u[k2].x * g[k2], u[k2].y * g[k2]);
        }
    }
    const int outs = W2 ? 2 : 1;
    const int nd = W2 && stream_dual_x(L) ? 2 : 1;  // outputs per round
    for (int w0 = 0; w0 < outs; w0 += nd) {
        __syncthreads();  // the spectrum is complete; the tables are free
        for (int i = cm.r0; i < nd * P; i += cm.rs) {
            const int t = i >= P ? 1 : 0, n1 = i - t * P, which = w0 + t;
            Cx<R> v[Q];
#pragma unroll
            for (int n2 = 0; n2 < Q; ++n2) v[n2] = line[n1 + P * n2];
            if (which)
#pragma unroll
                for (int n2 = 0; n2 < Q; ++n2) v[n2] = cmul_plain<R>(v[n2], ds[n1 + P * n2]);
            S::inv1(v, n1, tw, tab(t));
        }
        __syncthreads();
        for (int i = cm.r0; i < nd * Q; i += cm.rs) {
            const int t = i >= Q ? 1 : 0, k2 = i - t * Q, which = w0 + t;
            Cx<R> u[P];
            S::inv2(u, k2, tab(t));
            Cx<R>* out = which ? W2 : W;
#pragma unroll
            for (int k1 = 0; k1 < P / 2; ++k1) {
                const int x = k1 * Q + k2;
                if (live && x < nx) out[(size_t)x * ncol + col] = u[k1];
            }
        }
    }
}

// z forward (as zfwd_body): two charge rows per complex line, line c of the
// block's NC: rows y0 + 2c and y0 + 2c + 1 of plane x
template <typename R, int L>
__device__ __forceinline__ Cx<R>* zfwd_stream(R* __restrict__ q, const long long* __restrict__ qfix, int x, int y0,
                                              int ny, int nz, const Cx<R>* __restrict__ twg, int NC, const ScState* st,
                                              long long ncell) {
    using S = Steps<R, L>;
    constexpr int Q = S::Q, P = S::P, la = stream_la(L), lb = stream_lb<R>(L);
    extern __shared__ __align__(16) unsigned char smraw[];
    Cx<R>* tw = reinterpret_cast<Cx<R>*>(smraw);
    Cx<R>* A = tw + L;
    Cx<R>* B = A + NC * la;
    const float ufix = qfix ? st->qfix_inv : 0.f;
    load_twiddles<R>(tw, twg, L);
    __syncthreads();
    for (int i = threadIdx.x; i < NC * Q; i += blockDim.x) {
        const int c = i / Q, m = i - c * Q;
        const int ya = y0 + 2 * c, yb = ya + 1;
        Cx<R> v[P];
        const size_t ia0 = ((size_t)x * ny + ya) * nz + m;
        if (qfix) {
            long long fa[P / 2], fb[P / 2];
#pragma unroll
            for (int n1 = 0; n1 < P / 2; ++n1) {
                const bool in = n1 * Q + m < nz;
                const size_t ia = ia0 + n1 * Q;
                fa[n1] = (in && ya < ny && SC_IDX_OK(st, 21, ia, ncell)) ? qfix[ia] : 0;
                fb[n1] = (in && yb < ny && SC_IDX_OK(st, 22, ia + nz, ncell)) ? qfix[ia + nz] : 0;
            }
#pragma unroll
            for (int n1 = 0; n1 < P / 2; ++n1) {
                const bool in = n1 * Q + m < nz;
                const size_t ia = ia0 + n1 * Q;
                v[n1] = cx<R>((R)(__ll2float_rn(fa[n1]) * ufix), (R)(__ll2float_rn(fb[n1]) * ufix));
                if (in && ya < ny && SC_IDX_OK(st, 21, ia, ncell)) q[ia] = v[n1].x;
                if (in && yb < ny && SC_IDX_OK(st, 22, ia + nz, ncell)) q[ia + nz] = v[n1].y;
            }
        } else {
#pragma unroll
            for (int n1 = 0; n1 < P / 2; ++n1) {
                const bool in = n1 * Q + m < nz;
                const size_t ia = ia0 + n1 * Q;
                v[n1].x = (in && ya < ny && SC_IDX_OK(st, 21, ia, ncell)) ? q[ia] : (R)0;
                v[n1].y = (in && yb < ny && SC_IDX_OK(st, 22, ia + nz, ncell)) ? q[ia + nz] : (R)0;
            }
        }
        S::fwd1(v, m, tw, B + c * lb);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < NC * P; i += blockDim.x) {
        const int c = i / P, k1 = i - c * P;
        Cx<R> u[Q];
        S::fwd2(u, k1, B + c * lb);
#pragma unroll
        for (int k2 = 0; k2 < Q; ++k2) A[c * la + k1 + P * k2] = u[k2];
    }
    __syncthreads();
    return A;
}

}  // namespace ocsc
