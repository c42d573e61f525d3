// The FP64 convolution's separate passes for the two-step lengths
// (64 to 256 points), streamed and in block fixed point (sc_fx.cuh): a thread's
// inputs go from global memory into registers, the line's exponent is agreed on
// through shared memory, and the transform, the Green product and the inverse
// run in integers until the results are converted and stored.  Eight columns
// (z: NC lines) per block, 128 registers a thread and 512 threads' worth of blocks per SM so that one block's loads and
// barriers overlap the others' arithmetic.
//
// What bounds them: issue slots of the integer pipes (about half of them the
// conversions from and to double) and, at 64^3, one to two waves of blocks with
// five barriers.  Measured, double two-step -> these, 63^3 (128-point lines):
// x pass 82 -> 29 us, y forward 25 -> 12, y inverse 26 -> 10, z forward 16 -> 8,
// z inverse 20.6 -> 14.3; the kick of 200k particles 400 -> 316 us.
#pragma once
#include "sc_fft_dev.cuh"

namespace ocsc {

constexpr int FX_COLS = 8;
// Threads of a block of lines: of the wider step's items (Q per line) where there are
// few lines (z and Green passes, 2000 at 63^3: a round more would be exposed), of
// the narrower one's (P) in the x and y passes, where enough blocks stand beside
// each other and no warp should idle in the narrower step (x pass 31 -> 27 us, 29
// with its Green products under their own exponents, y 12 -> 9.6 and 10 -> 8.9, but Green
// passes 6.5 -> 9)
constexpr int fx_threads(int L) { return FX_COLS * two_step_q(L); }
constexpr int fx_threads_xy(int L) { return two_step_q(L) ? FX_COLS * (L / two_step_q(L)) : 0; }
// table of a line (odd stride), and dynamic shared memory of a pass over n lines
__host__ __device__ constexpr int fx_tab(int L) { return two_step_q(L) ? ((L / two_step_q(L)) * (two_step_q(L) + 1)) | 1 : 0; }
__host__ __device__ constexpr int fx_line(int L) { return L | 1; }
__host__ __device__ constexpr size_t fx_smem_cols(int L) { return sizeof(Fx2) * (size_t)(L + FX_COLS * fx_tab(L)); }
__host__ __device__ constexpr size_t fx_smem_z(int L, int NC) {
    return sizeof(Fx2) * (size_t)(L + NC * (fx_tab(L) + fx_line(L)));
}
__host__ __device__ constexpr size_t fx_smem_zi(int L, int NC) { return sizeof(Fx2) * (size_t)(L + NC * fx_tab(L)); }

// per-line words of a block: exponents and magnitudes
struct FxLines {
    int e[FX_COLS], m[3][FX_COLS];
};
static_assert(sizeof(FxLines) == 4 * FX_COLS * sizeof(int), "cleared word by word");
__device__ __forceinline__ void fx_clear(FxLines& s) {
    int* w = reinterpret_cast<int*>(&s);
    for (int i = threadIdx.x; i < (int)(sizeof(FxLines) / sizeof(int)); i += blockDim.x)
        w[i] = i < FX_COLS ? 1 : 0;  // e: 1, the exponent of denormals
}
// raise *word to v: the lanes of a warp that share a column (lane mod 8) first
__device__ __forceinline__ void fx_raise(int* word, int v) {
    v = max(v, __shfl_xor_sync(~0u, v, 8));
    v = max(v, __shfl_xor_sync(~0u, v, 16));
    if ((threadIdx.x & 31) < FX_COLS) atomicMax(word, v);
}
// the potential's largest exponent over a grid: every thread of the warp calls it
__device__ __forceinline__ void phi_raise(const ScState* st, int e) {
    e = __reduce_max_sync(~0u, e);
    if ((threadIdx.x & 31) == 0) atomicMax(&const_cast<ScState*>(st)->phi_exp, e);
}
template <int N>
__device__ __forceinline__ int fx_exp_of(const double2 (&d)[N]) {
    int e = 0;
#pragma unroll
    for (int n = 0; n < N; ++n) e = max(e, max(fx_exp(d[n].x), fx_exp(d[n].y)));
    return e;
}

// y pass, in place on W (as ypass_body): forward, rows < ny in, all L out;
// inverse, all in, rows < ny out
template <bool INV, int L>
__device__ __forceinline__ void ypass_fx(double2* __restrict__ W, int nx, int ny, int Kz,
                                         const double2* __restrict__ twg, VBlk vb) {
    using S = FxSteps<L>;
    constexpr int Q = S::Q, P = S::P;
    constexpr int A = INV ? P : Q, NIN = INV ? Q : P / 2;   // first step: items, inputs of one
    constexpr int B = INV ? Q : P, NOUT = INV ? P / 2 : Q;  // second step: items, outputs of one
    constexpr int RA = (A + P - 1) / P, RB = (B + P - 1) / P;  // rounds
    constexpr int BIT = INV ? S::B_INV : S::B_HALF;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ FxLines ln;
    FxW* tw = reinterpret_cast<FxW*>(smraw);
    const int kk = threadIdx.x & (FX_COLS - 1), m0 = threadIdx.x / FX_COLS;
    Fx2* tab = reinterpret_cast<Fx2*>(tw + L) + kk * fx_tab(L);
    const int col = vb.x * FX_COLS + kk;
    const bool live = col < nx * Kz;
    const int x = col / Kz, k = col - x * Kz;
    double2* line = W + (size_t)x * L * Kz + k;  // element y of the column at line[y * Kz]
    double2 d[RA][NIN];
    int e = 0;
#pragma unroll
    for (int r = 0; r < RA; ++r)
#pragma unroll
        for (int n = 0; n < NIN; ++n) {
            const int m = m0 + r * P, y = n * A + m;
            d[r][n] = (m < A && live && (INV || y < ny)) ? line[(size_t)y * Kz] : make_double2(0, 0);
        }
    fx_clear(ln);
    load_twiddles<double>(reinterpret_cast<double2*>(tw), twg, L);
#pragma unroll
    for (int r = 0; r < RA; ++r) e = max(e, fx_exp_of(d[r]));
    __syncthreads();
    fx_raise(&ln.e[kk], e);
    __syncthreads();
    const int E = ln.e[kk];
    unsigned mag = 0;
#pragma unroll
    for (int r = 0; r < RA; ++r) {
        const int m = m0 + r * P;
        if (m >= A) break;
        Fx2 v[INV ? Q : P];
#pragma unroll
        for (int n = 0; n < NIN; ++n) v[n] = cx<Fx>(fx_from<BIT>(d[r][n].x, E), fx_from<BIT>(d[r][n].y, E));
        if constexpr (INV) mag = max(mag, S::t_first(v, m, tw, tab));
        else mag = max(mag, S::template first<false, HALF_IN>(v, m, tw, tab));
    }
    fx_raise(&ln.m[0][kk], (int)mag);
    __syncthreads();
    const int sh = fx_room<INV ? P : Q>((unsigned)ln.m[0][kk]);
    const FxOut o(E, BIT - sh);
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        const int m = m0 + r * P;
        if (m >= B) break;
        Fx2 u[INV ? P : Q];
        if constexpr (INV) S::t_second(u, m, tab, sh);
        else S::template second<false>(u, m, tab, sh);
#pragma unroll
        for (int n = 0; n < NOUT; ++n) {
            const int y = n * B + m;
            if (live && (!INV || y < ny)) line[(size_t)y * Kz] = make_double2(fx_to(u[n].x, o), fx_to(u[n].y, o));
        }
    }
}

// x pass (as xconv_body): forward over the nx planes, Green multiply, inverse.
// The thread that holds X[k1 + P k2] after the forward transform is the one
// that starts the inverse with them, so the spectrum never leaves its registers;
// the Green entries of a line are integers under one exponent too
template <int L>
__device__ __forceinline__ void xconv_fx(double2* __restrict__ W, const double* __restrict__ G, int nx, int My, int Kz,
                                         int Ky, const double2* __restrict__ twg, const ScState* st, VBlk vb) {
    using S = FxSteps<L>;
    constexpr int Q = S::Q, P = S::P;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ FxLines ln;
    FxW* tw = reinterpret_cast<FxW*>(smraw);
    constexpr int RQ = (Q + P - 1) / P;  // rounds of the Q-item steps
    const int kk = threadIdx.x & (FX_COLS - 1), m = threadIdx.x / FX_COLS;
    Fx2* tab = reinterpret_cast<Fx2*>(tw + L) + kk * fx_tab(L);
    const int col = vb.x * FX_COLS + kk;
    const int ncol = My * Kz;
    const bool live = col < ncol;
    const int ky = col / Kz, k = col - ky * Kz;
    const int gy = ky <= My - ky ? ky : My - ky;
    const int gk = gy * Kz + k;  // the column's Green entry at gx * Ky * Kz + gk
    const int KyKz = Ky * Kz;
    int E;
    unsigned mag = 0;
    {
        double2 d[RQ][P / 2];
#pragma unroll
        for (int r = 0; r < RQ; ++r)
#pragma unroll
            for (int n1 = 0; n1 < P / 2; ++n1) {
                const int x = n1 * Q + m + r * P;
                d[r][n1] = (m + r * P < Q && x < nx && live) ? W[(size_t)x * ncol + col] : make_double2(0, 0);
            }
        fx_clear(ln);
        load_twiddles<double>(reinterpret_cast<double2*>(tw), twg, L);
        int e = 0;
#pragma unroll
        for (int r = 0; r < RQ; ++r) e = max(e, fx_exp_of(d[r]));
        __syncthreads();
        fx_raise(&ln.e[kk], e);
        __syncthreads();
        E = ln.e[kk];
#pragma unroll
        for (int r = 0; r < RQ; ++r) {
            if (m + r * P >= Q) break;
            Fx2 v[P];
#pragma unroll
            for (int n1 = 0; n1 < P / 2; ++n1)
                v[n1] = cx<Fx>(fx_from<S::B_HALF>(d[r][n1].x, E), fx_from<S::B_HALF>(d[r][n1].y, E));
            mag = max(mag, S::template first<false, HALF_IN>(v, m + r * P, tw, tab));
        }
    }
    double g[Q];
#pragma unroll
    for (int k2 = 0; k2 < Q; ++k2) {
        const int kx = m + P * k2, gx = kx <= L - kx ? kx : L - kx;
        const long long gi = (long long)gx * KyKz + gk;
        g[k2] = (live && SC_IDX_OK(st, 23, gi, (long long)(L / 2 + 1) * KyKz)) ? G[gi] : 0.0;
    }
    fx_raise(&ln.m[0][kk], (int)mag);
    __syncthreads();
    Fx2 u[Q];
    int top = 0;
    int sh = fx_room<Q>((unsigned)ln.m[0][kk]);
    int bit = S::B_HALF - sh;  // the bit of 2^E in what is held
    S::template second<false>(u, m, tab, sh);
    // the row of the table that this thread has just read holds its exponents
    // until its products' shifts are known (16 registers less, 26 spilled)
    Fx2* row = tab + m * S::ROW;
#pragma unroll
    for (int k2 = 0; k2 < Q; ++k2) {
        int e;
        const FxC c = fx_fraction(g[k2], e);
        u[k2] = cx<Fx>(fx_mul(u[k2].x, c), fx_mul(u[k2].y, c));
        top = max(top, fx_top(u[k2], e));
        row[k2].x.v = e;
    }
    // value = held * 2^(E - 1023 - bit) * 2^(eg - 1022)
    fx_raise(&ln.m[1][kk], top);
    __syncthreads();
    const int EG = ln.m[1][kk] - (fx_bit(Q) + 1);  // the exponent that leaves the largest its room
    bit -= EG - 1022;
#pragma unroll
    for (int k2 = 0; k2 < Q; ++k2) u[k2] = fx_scale(u[k2], EG - (int)row[k2].x.v);
    mag = S::t_first(u, m, tw, tab);  // over the row of the table that this thread has read
    fx_raise(&ln.m[2][kk], (int)mag);
    __syncthreads();
    sh = fx_room<P>((unsigned)ln.m[2][kk]);
    const FxOut o(EG > 2 * FX_BAD ? FX_BAD : E, bit - sh);
#pragma unroll
    for (int r = 0; r < RQ; ++r) {
        const int k2 = m + r * P;
        if (k2 >= Q) break;
        Fx2 w[P];
        S::t_second(w, k2, tab, sh);
#pragma unroll
        for (int k1 = 0; k1 < P / 2; ++k1) {
            const int x = k1 * Q + k2;
            if (live && x < nx) W[(size_t)x * ncol + col] = make_double2(fx_to(w[k1].x, o), fx_to(w[k1].y, o));
        }
    }
}

// z forward (as zfwd_body, the unpacking of the two rows in double as there): line
// c of the block's NC: charge rows y0 + 2c and y0 + 2c + 1 of plane x
template <int L>
__device__ __forceinline__ void zfwd_fx(const double* __restrict__ q, double2* __restrict__ W, int ny, int nz, int My,
                                        int Kz, const double2* __restrict__ twg, int NC, const ScState* st, VBlk vb) {
    using S = FxSteps<L>;
    constexpr int Q = S::Q, P = S::P;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ FxLines ln;
    FxW* tw = reinterpret_cast<FxW*>(smraw);
    double2* spec = reinterpret_cast<double2*>(tw + L);
    Fx2* tabs = reinterpret_cast<Fx2*>(spec + NC * fx_line(L));
    const int x = vb.y, y0 = vb.x * 2 * NC;
    const long long ncell = (long long)vb.ny * ny * nz;
    (void)ncell;  // read by the index checks of checked builds
    const int c = threadIdx.x / Q, m = threadIdx.x - c * Q;  // blockDim = NC Q
    const int ra = y0 + 2 * c, rb = ra + 1;
    double2 d[P / 2];
#pragma unroll
    for (int n1 = 0; n1 < P / 2; ++n1) {
        const int z = n1 * Q + m;
        const size_t i = ((size_t)x * ny + ra) * nz + z;
        d[n1].x = (z < nz && ra < ny && SC_IDX_OK(st, 21, i, ncell)) ? q[i] : 0.0;
        d[n1].y = (z < nz && rb < ny && SC_IDX_OK(st, 22, i + nz, ncell)) ? q[i + nz] : 0.0;
    }
    fx_clear(ln);
    load_twiddles<double>(reinterpret_cast<double2*>(tw), twg, L);
    __syncthreads();
    atomicMax(&ln.e[c], fx_exp_of(d));
    __syncthreads();
    {
        const int E = ln.e[c];
        Fx2 v[P];
#pragma unroll
        for (int n1 = 0; n1 < P / 2; ++n1)
            v[n1] = cx<Fx>(fx_from<S::B_HALF>(d[n1].x, E), fx_from<S::B_HALF>(d[n1].y, E));
        atomicMax(&ln.m[0][c], (int)S::template first<false, HALF_IN>(v, m, tw, tabs + c * fx_tab(L)));
    }
    __syncthreads();
    if (m < P) {
        Fx2 u[Q];
        const int sh = fx_room<Q>((unsigned)ln.m[0][c]);
        const FxOut o(ln.e[c], S::B_HALF - sh);
        S::template second<false>(u, m, tabs + c * fx_tab(L), sh);
#pragma unroll
        for (int k2 = 0; k2 < Q; ++k2)
            spec[c * fx_line(L) + m + P * k2] = make_double2(fx_to(u[k2].x, o), fx_to(u[k2].y, o));
    }
    __syncthreads();
    for (DivWalk w(threadIdx.x, blockDim.x, Kz); w.q < NC; w.next()) {
        const int l = w.q, k = w.r, ya = y0 + 2 * l, yb = ya + 1;
        const double2 Z = spec[l * fx_line(L) + k], Zm = spec[l * fx_line(L) + (k == 0 ? 0 : L - k)];
        if (!SC_IDX_OK(st, 24, ((long long)x * My + (yb < ny ? yb : ya)) * Kz + k, (long long)vb.ny * My * Kz)) continue;
        // the halving rides on the potential's scale (unpack_half)
        if (ya < ny) W[((size_t)x * My + ya) * Kz + k] = make_double2(Z.x + Zm.x, Z.y - Zm.y);
        if (yb < ny) W[((size_t)x * My + yb) * Kz + k] = make_double2(Z.y + Zm.y, Zm.x - Z.x);
    }
}

// z inverse (as zinv_body): two rows per complex line, Z = A + iB Hermitian-extended
// above L / 2 (that sum in double, as there), out(v) scales a value of the potential
template <int L, typename Out>
__device__ __forceinline__ void zinv_fx(const double2* __restrict__ W, double* __restrict__ phi, int ny, int nz, int My,
                                        int Kz, const double2* __restrict__ twg, int NC, Out out, const ScState* st,
                                        VBlk vb) {
    using S = FxSteps<L>;
    constexpr int Q = S::Q, P = S::P;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ FxLines ln;
    FxW* tw = reinterpret_cast<FxW*>(smraw);
    const int x = vb.y, y0 = vb.x * 2 * NC;
    const int c = threadIdx.x / Q, m = threadIdx.x - c * Q;  // blockDim = NC Q
    Fx2* tab = reinterpret_cast<Fx2*>(tw + L) + c * fx_tab(L);
    const int ra = y0 + 2 * c, rb = ra + 1;
    const double2* Wa = W + ((size_t)x * My + ra) * Kz;
    const bool la = m < P && ra < ny, lb = m < P && rb < ny;
    double2 d[Q];
    constexpr int U = 4;  // entries per round: their loads are issued together
#pragma unroll
    for (int n0 = 0; n0 < Q; n0 += U) {
        double2 a[U], b[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = m + P * (n0 + u), kk = k < Kz ? k : L - k;
            a[u] = la ? Wa[kk] : make_double2(0, 0);
            b[u] = lb ? Wa[Kz + kk] : make_double2(0, 0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = m + P * (n0 + u);
            d[n0 + u] = k < Kz ? make_double2(a[u].x - b[u].y, a[u].y + b[u].x)
                               : make_double2(a[u].x + b[u].y, b[u].x - a[u].y);
        }
    }
    fx_clear(ln);
    load_twiddles<double>(reinterpret_cast<double2*>(tw), twg, L);
    __syncthreads();
    if (m < P) atomicMax(&ln.e[c], fx_exp_of(d));
    __syncthreads();
    const int E = ln.e[c];
    if (m < P) {
        Fx2 v[Q];
#pragma unroll
        for (int n = 0; n < Q; ++n) v[n] = cx<Fx>(fx_from<S::B_INV>(d[n].x, E), fx_from<S::B_INV>(d[n].y, E));
        atomicMax(&ln.m[0][c], (int)S::t_first(v, m, tw, tab));
    }
    __syncthreads();
    const int sh = fx_room<P>((unsigned)ln.m[0][c]);
    const FxOut o(E, S::B_INV - sh);
    Fx2 u[P];
    S::t_second(u, m, tab, sh);
    int e = 0;
#pragma unroll
    for (int k1 = 0; k1 < P / 2; ++k1) {
        const int z = k1 * Q + m;
        double* p = phi + ((size_t)x * ny + ra) * nz + z;
        auto put = [&](double* dst, double v) {
            *dst = v;
            e = max(e, fx_exp(v));
        };
        if (z < nz && ra < ny) put(p, out(fx_to(u[k1].x, o)));
        if (z < nz && rb < ny) put(p + nz, out(fx_to(u[k1].y, o)));
    }
    phi_raise(st, e);
}

// Forward transform of one even line pair per line (the Green passes): item m of
// line c reads ld(n), n = Q n1 + m, and the outputs k <= L / 2 go to st(k, value)
template <int L, typename Load, typename Store>
__device__ __forceinline__ void even_fx(int c, int m, const double2* __restrict__ twg, Load&& ld, Store&& put) {
    using S = FxSteps<L>;
    constexpr int Q = S::Q, P = S::P;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ FxLines ln;
    FxW* tw = reinterpret_cast<FxW*>(smraw);
    Fx2* tab = reinterpret_cast<Fx2*>(tw + L) + c * fx_tab(L);
    double2 d[P];
#pragma unroll
    for (int n1 = 0; n1 < P; ++n1) d[n1] = ld(n1 * Q + m);
    fx_clear(ln);
    load_twiddles<double>(reinterpret_cast<double2*>(tw), twg, L);
    __syncthreads();
    atomicMax(&ln.e[c], fx_exp_of(d));
    __syncthreads();
    const int E = ln.e[c];
    {
        Fx2 v[P];
#pragma unroll
        for (int n1 = 0; n1 < P; ++n1) v[n1] = cx<Fx>(fx_from<S::B_FULL>(d[n1].x, E), fx_from<S::B_FULL>(d[n1].y, E));
        atomicMax(&ln.m[0][c], (int)S::template first<false, DFT_FULL>(v, m, tw, tab));
    }
    __syncthreads();
    if (m < P) {
        const int sh = fx_room<Q>((unsigned)ln.m[0][c]);
        const FxOut o(E, S::B_FULL - sh);
        Fx2 u[Q];
        S::template second<false>(u, m, tab, sh);
#pragma unroll
        for (int k2 = 0; k2 <= Q / 2; ++k2) {
            const int k = m + P * k2;
            if (k <= L / 2) put(k, make_double2(fx_to(u[k2].x, o), fx_to(u[k2].y, o)));
        }
    }
}

}  // namespace ocsc
