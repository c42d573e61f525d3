// Free-space potential by zero-padded FFT convolution with the integrated
// Green's function, and the forward-difference field grids.
//
// Restates SpaceCharge.potential (ocelot/cpbd/sc.py:135-168) and the field
// grids of el_field (sc.py:195-200).  The reference convolves on a
// (2N-1)^3 complex grid; the linear convolution is the same on any padded
// length M >= 2N-1, so each axis is padded to a length with a 2/4/8 radix
// plan.  Only the N^3 octant of the charge is non-zero and only the N^3
// octant of the result is kept, so the passes skip the zero planes:
//
//   F1  z: real-to-complex of the nx*ny charge lines (two lines per complex FFT)
//   F2  y: forward FFT of the nx*Kz columns, zero-padded from ny to My
//   F3  x: forward FFT, multiply by the real Green spectrum, inverse FFT,
//          keep x < nx (the only pass that sees all Mx planes, in shared memory)
//   B2  y: inverse FFT, keep y < ny
//   B1  z: complex-to-real of the nx*ny lines, keep z < nz, scale by
//          1/(Mx*My*Mz) and 1/(4*pi*eps0*hx*hy*hz)
//
// The complex work grid W[x][y][kz] (x < nx, y < My, kz <= Mz/2) stays in
// HBM/L2 between passes.  Lines of 64 to 256 points take two register steps,
// streamed from and to global memory (sc_fft_stream.cuh in FP32, in 64-bit block
// fixed point for FP64, sc_fft_fx.cuh); other lengths stage whole lines in
// shared memory (sc_fft_dev.cuh).
#include "sc_common.cuh"
#include "sc_fft_dev.cuh"
#include "sc_fft_stream.cuh"
#include "sc_fft_fx.cuh"

namespace ocsc {

// threads of the staged passes (the lengths outside the two-step form)
template <typename R>
constexpr int FFT_THREADS = sizeof(R) == 8 ? 128 : 256;
constexpr int FFT_MINB = 4;
// the fixed-point passes: 128 registers
constexpr int FX_MINB(int L) { return 512 / fx_threads(L); }
constexpr int FX_MINB_XY(int L) { return 512 / fx_threads_xy(L); }

// complex lines (two real lines each) per block of the z passes: up to 8,
// so that a 64^3 mesh gives 256 blocks
static inline int z_lines_per_block(int Mz) {
    int nc = 1024 / Mz;
    return nc < 1 ? 1 : (nc > 8 ? 8 : nc);
}
// the fixed-point z passes: whole warps of two_step_q(Mz) threads a line.  Eight lines
// a block against four, forward + inverse (us): 48^3 16.8 / 17.5, 63^3 25.0 / 24.9, 96^3
// 51.7 / 54.9; at 256 points the other way, 100 x 100 x 120 94 / 89
template <typename R>
static inline int z_lines(int Mz) {
    const int nc = z_lines_per_block(Mz);
    return sizeof(R) == 8 && uses_two_step(Mz) ? (Mz > 192 ? 4 : 8) : nc;
}
// columns per block in the strided passes: 16, fewer when two line buffers
// of 16 columns would not fit in shared memory (FP64 at M = 512)
template <typename R>
static inline int strided_cols(int M, int nbuf = 2) {
    int tk = sizeof(R) == 8 && M > 64 ? 8 : 16;
    while (tk > 2 && sizeof(Cx<R>) * (size_t)(M + nbuf * tk * fft_ls(M)) > 200 * 1024) tk /= 2;
    return tk;
}
// dynamic shared memory of the separate passes over lines of length M: the
// streamed form's twiddles, difference factors, tables and lines
// (sc_fft_stream.cuh), else twiddles and whole line buffers
template <typename R>
static inline size_t smem_zf(int M, int NC) {
    if (sizeof(R) == 8 && uses_two_step(M)) return fx_smem_z(M, NC);
    return sizeof(Cx<R>) * (streamed<R>(M) ? M + NC * (size_t)(stream_la(M) + stream_lb<R>(M))
                                                : M + 2 * NC * (size_t)fft_ls(M));
}
template <typename R>
static inline size_t smem_zi(int M, int NC) {
    if (sizeof(R) == 8 && uses_two_step(M)) return fx_smem_zi(M, NC);
    return sizeof(Cx<R>) * (M + 2 * NC * (size_t)fft_ls(M));
}
template <typename R>
static inline size_t smem_yf(int M, int TK) {
    if (sizeof(R) == 8 && uses_two_step(M)) return fx_smem_cols(M);
    return sizeof(Cx<R>) * (streamed<R>(M) ? M + TK * (size_t)stream_lb<R>(M) : M + 2 * TK * (size_t)fft_ls(M));
}
template <typename R>
static inline size_t smem_yi(int M, int TK, bool w3) {
    if (sizeof(R) == 8 && uses_two_step(M)) return fx_smem_cols(M);
    return sizeof(Cx<R>) * (streamed<R>(M) ? (w3 ? 2 : 1) * (M + TK * (size_t)stream_lb<R>(M))
                                                : M + (w3 ? 3 : 2) * TK * (size_t)fft_ls(M));
}
template <typename R>
static inline size_t smem_x(int M, int TK, bool w2) {
    if (sizeof(R) == 8 && uses_two_step(M)) return fx_smem_cols(M);
    return sizeof(Cx<R>) * (streamed<R>(M)
                                ? (w2 ? 2 : 1) * M + TK * (size_t)(stream_la(M) +
                                                                   (w2 && stream_dual_x(M) ? 2 : 1) * stream_lb<R>(M))
                                : M + (w2 ? 3 : 2) * TK * (size_t)fft_ls(M));
}
// the plan's columns per block (SC_PARAM_FFT_COLS_X / _Y; 0: strided_cols),
// never more than fit.  The columns are independent lines, so the grouping
// changes no result.
template <typename R>
static inline int pass_cols(int want, int M, int nbuf = 2) {
    if (sizeof(R) == 8 && uses_two_step(M)) return FX_COLS;
    const int fit = strided_cols<R>(M, nbuf);
    return (want > 0 && want < fit) ? want : fit;
}

// Spectral fields (FP32 with SC_FP32_SPECTRAL_FIELDS).  The field grids are
// forward differences of the potential, Ex[i] = (phi[i] - phi[i+1]) / hx
// (sc.py:195-200); on the padded grid that difference is the product of the
// spectrum with D(k) = 1 - exp(2 pi i k / M), exact for every cell the
// reference keeps.  Taking it in Fourier space before the inverse transforms
// makes the rounding of each field relative to the field itself instead of
// to the potential, which is hundreds of times larger than the differences
// of neighbouring cells.
//   Ex: x inverse of (spectrum x D(kx)) into W2, then y and z inverses
//   Ey: y inverse of (W x D(ky)) into W3 (W after the x inverse), then z
//   Ez: z inverse of (y-inverted W) x D(kz)
// The potential itself is kept (z inverse of the y-inverted W).
template <typename R>
struct Spec {
    Cx<R>* W2;                       // the x-differenced grid (Ex); nullptr: no spectral fields
    Cx<R>* W3;                       // the y-differenced grid (Ey), separate passes only
    const Cx<R>* dx;                 // D(k) per axis
    const Cx<R>* dy;
    const Cx<R>* dz;
    R* ex;                           // field grids [nx][ny][nz], zero on their last plane
    R* ey;
    R* ez;
    int f0;                          // first output of the inverse passes: 0 with the potential, 1 without
};
template <typename R>
__device__ __forceinline__ Cx<R> cmul(Cx<R> a, Cx<R> b) {
    return cx<R>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// Unpacking two real lines from one complex transform halves their sums; in
// FP64 that factor rides on the potential's scale instead (out_scale64; a power
// of two, so the same bits), four FP64 instructions per spectrum entry fewer.
template <typename R>
__device__ __forceinline__ constexpr R unpack_half() { return sizeof(R) == 8 ? (R)1 : (R)0.5; }
template <typename R>
__device__ __forceinline__ Cx<R> scaled(R re, R im, R h) {
    if constexpr (sizeof(R) == 8) return cx<R>(re, im);
    else return cx<R>(re * h, im * h);
}
// FP64 output: v / M / (4 pi eps0 hx hy hz) (sc.py:164-167); the division by
// its reciprocal with one correction (correctly rounded up to the last bit's
// ties), three instructions instead of the IEEE form's dozen
struct OutScale64 {
    double norm, denom, rdenom;
    __device__ __forceinline__ double operator()(double v) const {
        const double a = v * norm, q = a * rdenom;
        return fma(fma(-q, denom, a), rdenom, q);
    }
};
__device__ __forceinline__ OutScale64 out_scale64(const ScState* st) {
    return OutScale64{0.5 * st->phi_norm, st->phi_denom, __drcp_rn(st->phi_denom)};
}

// Stage the charge of NC complex z lines into the line buffer a (line c at
// a + c * lz): the real part of line c is row y0 + 2c of plane x, the
// imaginary part row y0 + 2c + 1, zero-padded from nz to Mz.  With qfix the
// charge arrives as the 64-bit fixed-point grid, is scaled to R and is also
// stored in q.  U elements per thread per round: all their loads are issued
// before any of them is converted or stored, one memory round trip per round.
// code, code + 1: the index-check codes of the two rows
template <typename R>
__device__ __forceinline__ void stage_charge_lines(R* __restrict__ q, const long long* __restrict__ qfix,
                                                   Cx<R>* __restrict__ a, int lz, int x, int y0, int NC, int ny,
                                                   int nz, int Mz, const ScState* st, long long ncell, int code) {
    constexpr int U = 4;
    const float ufix = qfix ? st->qfix_inv : 0.f;
    for (DivWalk w(threadIdx.x, blockDim.x, Mz); w.q < NC;) {
        int cs[U], zs[U];
        bool oka[U], okb[U];
        size_t ia[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            cs[u] = w.q;
            zs[u] = w.r;
            w.next();
            const int ya = y0 + 2 * cs[u], yb = ya + 1;
            const bool in = cs[u] < NC && zs[u] < nz;
            ia[u] = ((size_t)x * ny + ya) * nz + zs[u];
            oka[u] = in && ya < ny && SC_IDX_OK(st, code, ia[u], ncell);
            okb[u] = in && yb < ny && SC_IDX_OK(st, code + 1, ia[u] + nz, ncell);
        }
        R re[U], im[U];
        if (qfix) {
            long long fa[U], fb[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                fa[u] = oka[u] ? qfix[ia[u]] : 0;
                fb[u] = okb[u] ? qfix[ia[u] + nz] : 0;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                re[u] = (R)(__ll2float_rn(fa[u]) * ufix);
                im[u] = (R)(__ll2float_rn(fb[u]) * ufix);
                if (oka[u]) q[ia[u]] = re[u];
                if (okb[u]) q[ia[u] + nz] = im[u];
            }
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                re[u] = oka[u] ? q[ia[u]] : (R)0;
                im[u] = okb[u] ? q[ia[u] + nz] : (R)0;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (cs[u] < NC) a[cs[u] * lz + zs[u]] = cx<R>(re[u], im[u]);
    }
}

// qfix != nullptr: the charge arrives as the 64-bit fixed-point grid of the
// FP32 form's exact deposit; it is scaled to R here and also stored in q
// (the charge grid an inspection reads back).
//
// STREAM: what the body's lines take -- ST_NO staged passes (any length), ST_ANY
// by the length at run time (the batched kernels), a length the streamed pass
// of that length.  The separate FP32 passes have a kernel per streamed length, with
// as many threads as the length has items for 16 columns: a 64-point pass in blocks
// of 256 leaves half of them idle in each step (32^3: z 5.4 -> 3.6 us, y 5.8 -> 2.5,
// x 9.0 -> 3.9), and a shared kernel takes the registers of its longest line
enum { ST_NO = 0, ST_ANY = -1 };
template <typename R, int STREAM, typename F>
__device__ __forceinline__ bool stream_pass(int L, F&& f) {
    if constexpr (STREAM > 0) {
        f(IntC<STREAM>{});
        return true;
    } else if constexpr (STREAM == ST_ANY) {
        return with_stream<R>(L, f);
    } else {
        return false;
    }
}

template <typename R, int STREAM>
__device__ __forceinline__ void zfwd_body(R* __restrict__ q, const long long* __restrict__ qfix,
                                          Cx<R>* __restrict__ W, int ny, int nz, int My, int Kz,
                                          const RadixPlan& rz, const Cx<R>* __restrict__ twg, int NC,
                                          const ScState* st, VBlk vb) {
    extern __shared__ __align__(16) unsigned char smraw[];
    if (st->status) return;
    const int Mz = rz.L;
    const int x = vb.y;
    const int y0 = vb.x * 2 * NC;
    Cx<R>* res = nullptr;
    int lz = stream_la(Mz);
    if (!stream_pass<R, STREAM>(Mz, [&](auto L) {
            res = zfwd_stream<R, decltype(L)::value>(q, qfix, x, y0, ny, nz, twg, NC, st, (long long)vb.ny * ny * nz);
        })) {
        lz = fft_ls(Mz);
        Cx<R>* tw = reinterpret_cast<Cx<R>*>(smraw);
        Cx<R>* a = tw + Mz;
        Cx<R>* b = a + NC * lz;
        load_twiddles<R>(tw, twg, Mz);
        stage_charge_lines<R>(q, qfix, a, lz, x, y0, NC, ny, nz, Mz, st, (long long)vb.ny * ny * nz, 21);
        __syncthreads();
        res = fft_lines<R, false, true, false>(a, b, lz, NC, rz, tw);
    }
    for (DivWalk w(threadIdx.x, blockDim.x, Kz); w.q < NC; w.next()) {
        const int c = w.q, k = w.r;
        const int ya = y0 + 2 * c, yb = ya + 1;
        const Cx<R> Z = res[c * lz + k];
        const Cx<R> Zm = res[c * lz + (k == 0 ? 0 : Mz - k)];
        const R h = unpack_half<R>();
        if (!SC_IDX_OK(st, 24, ((long long)x * My + (yb < ny ? yb : ya)) * Kz + k, (long long)vb.ny * My * Kz)) continue;
        if (ya < ny) W[((size_t)x * My + ya) * Kz + k] = scaled<R>(Z.x + Zm.x, Z.y - Zm.y, h);
        if (yb < ny) W[((size_t)x * My + yb) * Kz + k] = scaled<R>(Z.y + Zm.y, Zm.x - Z.x, h);
    }
}

template <typename R>
__global__ void __launch_bounds__(FFT_THREADS<R>, FFT_MINB) k_zfwd(R* __restrict__ q, const long long* __restrict__ qfix,
                                                      Cx<R>* __restrict__ W, int ny, int nz, int My, int Kz,
                                                      RadixPlan rz, const Cx<R>* __restrict__ twg, int NC,
                                                      const ScState* st) {
    pdl_wait();
    zfwd_body<R, ST_NO>(q, qfix, W, ny, nz, My, Kz, rz, twg, NC, st, hw_vblk());
}
template <int L>
__global__ void __launch_bounds__(128, 8) k_zfwd_s(float* __restrict__ q, const long long* __restrict__ qfix,
                                                   Cx<float>* __restrict__ W, int ny, int nz, int My, int Kz,
                                                   RadixPlan rz, const Cx<float>* __restrict__ twg, int NC,
                                                   const ScState* st) {
    pdl_wait();
    zfwd_body<float, L>(q, qfix, W, ny, nz, My, Kz, rz, twg, NC, st, hw_vblk());
}

template <int L>
__global__ void __launch_bounds__(fx_threads(L), FX_MINB(L)) k_zfwd_fx(double* __restrict__ q, double2* __restrict__ W,
                                                                    int ny, int nz, int My, int Kz,
                                                                    const double2* __restrict__ twg, int NC,
                                                                    const ScState* st) {
    pdl_wait();
    if (st->status) return;
    zfwd_fx<L>(q, W, ny, nz, My, Kz, twg, NC, st, hw_vblk());
}
template <bool INV, int L>
__global__ void __launch_bounds__(fx_threads_xy(L), FX_MINB_XY(L)) k_ypass_fx(double2* __restrict__ W, int nx, int ny, int Kz,
                                                                     const double2* __restrict__ twg,
                                                                     const ScState* st) {
    pdl_wait();
    if (st->status) return;
    ypass_fx<INV, L>(W, nx, ny, Kz, twg, hw_vblk());
}
template <int L>
__global__ void __launch_bounds__(fx_threads_xy(L), FX_MINB_XY(L)) k_xconv_fx(double2* __restrict__ W,
                                                                     const double* __restrict__ G, int nx, int My,
                                                                     int Kz, int Ky, const double2* __restrict__ twg,
                                                                     const ScState* st) {
    pdl_wait();
    if (st->status) return;
    xconv_fx<L>(W, G, nx, My, Kz, Ky, twg, st, hw_vblk());
}

// strided pass along y: forward (rows < ny in, all My out) or inverse (all in, rows < ny out),
// in place on W.  The columns are the nx * Kz lines (x, kz), flattened as
// x * Kz + kz; block vb.x takes TK consecutive ones (a block may straddle two
// x planes).  W3 != nullptr (inverse, spectral fields): the block also
// transforms its columns of W multiplied by D(ky) into W3 (a third line buffer)
template <typename R, bool INV, int STREAM>
__device__ __forceinline__ void ypass_body(Cx<R>* __restrict__ W, int nx, int ny, int My, int Kz, const RadixPlan& ry,
                                           const Cx<R>* __restrict__ twg, int TK, const ScState* st, VBlk vb,
                                           Cx<R>* __restrict__ W3 = nullptr, const Cx<R>* __restrict__ dy = nullptr) {
    extern __shared__ __align__(16) unsigned char smraw[];
    if (st->status) return;
    if (stream_pass<R, STREAM>(My, [&](auto L) {
            ypass_stream<R, INV, decltype(L)::value>(W, nx, ny, Kz, twg, TK, vb, W3, dy);
        }))
        return;
    const int ls = fft_ls(My);
    Cx<R>* tw = reinterpret_cast<Cx<R>*>(smraw);
    Cx<R>* a = tw + My;
    Cx<R>* b = a + TK * ls;
    Cx<R>* c = b + TK * ls;
    load_twiddles<R>(tw, twg, My);
    const ColMap cm(TK);
    const int col = vb.x * TK + cm.kk;
    const bool live = col < nx * Kz;
    const int x = col / Kz, k = col - x * Kz;
    const size_t base = ((size_t)x * My) * Kz + k;  // element y of the column at base + y * Kz
    const int nin = INV ? My : ny;
    Cx<R>* la = a + cm.kk * ls;
    Cx<R>* lc = c + cm.kk * ls;
    constexpr int U = 8;  // rows per round: their loads are issued together
    for (int y0 = cm.r0; y0 < My; y0 += U * cm.rs) {
        Cx<R> v[U], d[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int y = y0 + u * cm.rs;
            v[u] = (y < nin && live) ? W[base + (size_t)y * Kz] : cx<R>(0, 0);
            d[u] = (W3 && y < My) ? dy[y] : cx<R>(0, 0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int y = y0 + u * cm.rs;
            if (y < My) {
                la[y] = v[u];
                if (W3) lc[y] = cmul(v[u], d[u]);
            }
        }
    }
    __syncthreads();
    Cx<R>* res = fft_lines<R, INV, true, false>(a, b, ls, TK, ry, tw);
    const int nout = INV ? ny : My;
    if (live)
        for (int y = cm.r0; y < nout; y += cm.rs) W[base + (size_t)y * Kz] = res[cm.kk * ls + y];
    if (W3) {
        __syncthreads();  // a and b are free
        Cx<R>* res3 = fft_lines<R, INV, true, false>(c, a, ls, TK, ry, tw);
        if (live)
            for (int y = cm.r0; y < nout; y += cm.rs) W3[base + (size_t)y * Kz] = res3[cm.kk * ls + y];
    }
}

// blockIdx.y = 0: W (and, with spectral fields, W x D(ky) into W3);
// blockIdx.y = 1 (inverse, spectral fields): the x-differenced grid W2 in place
template <typename R, bool INV>
__global__ void __launch_bounds__(FFT_THREADS<R>, FFT_MINB) k_ypass(Cx<R>* __restrict__ W, int nx, int ny, int My, int Kz,
                                                       RadixPlan ry, const Cx<R>* __restrict__ twg,
                                                       int TK, const ScState* st, Spec<R> sp) {
    pdl_wait();
    if (blockIdx.y == 0) ypass_body<R, INV, ST_NO>(W, nx, ny, My, Kz, ry, twg, TK, st, hw_vblk(), sp.W3, sp.dy);
    else ypass_body<R, INV, ST_NO>(sp.W2, nx, ny, My, Kz, ry, twg, TK, st, hw_vblk());
}
template <bool INV, int L>
__global__ void __launch_bounds__(stream_threads(L), stream_minb(L))
    k_ypass_s(Cx<float>* __restrict__ W, int nx, int ny, int My, int Kz, RadixPlan ry,
              const Cx<float>* __restrict__ twg, int TK, const ScState* st, Spec<float> sp) {
    pdl_wait();
    if (blockIdx.y == 0)
        ypass_body<float, INV, L>(W, nx, ny, My, Kz, ry, twg, TK, st, hw_vblk(), INV ? sp.W3 : nullptr, sp.dy);
    else ypass_body<float, INV, L>(sp.W2, nx, ny, My, Kz, ry, twg, TK, st, hw_vblk());
}

// x pass: forward FFT of the nx non-zero planes, Green multiply, inverse FFT, keep x < nx.
// The columns are the My * Kz lines (ky, kz), flattened as ky * Kz + kz (the
// element x of a column at x * My * Kz + column); block vb.x takes TK
// consecutive ones.  W2 != nullptr (spectral fields): the product times D(kx)
// goes through its own inverse transform (a third line buffer) into W2
template <typename R, int STREAM>
__device__ __forceinline__ void xconv_body(Cx<R>* __restrict__ W, const R* __restrict__ G, int nx, int My, int Kz,
                                           int Ky, const RadixPlan& rx, const Cx<R>* __restrict__ twg, int TK,
                                           const ScState* st, VBlk vb, Cx<R>* __restrict__ W2 = nullptr,
                                           const Cx<R>* __restrict__ dx = nullptr) {
    extern __shared__ __align__(16) unsigned char smraw[];
    if (st->status) return;
    const int Mx = rx.L;
    if (stream_pass<R, STREAM>(Mx, [&](auto L) {
            xconv_stream<R, decltype(L)::value>(W, G, nx, My, Kz, Ky, twg, TK, st, vb, W2, dx);
        }))
        return;
    const int ls = fft_ls(Mx);
    Cx<R>* tw = reinterpret_cast<Cx<R>*>(smraw);
    Cx<R>* a = tw + Mx;
    Cx<R>* b = a + TK * ls;
    Cx<R>* c = b + TK * ls;
    load_twiddles<R>(tw, twg, Mx);
    const ColMap cm(TK);
    const int col = vb.x * TK + cm.kk;
    const int ncol = My * Kz;
    const bool live = col < ncol;
    const int ky = col / Kz, k = col - ky * Kz;
    const int gy = ky <= My - ky ? ky : My - ky;
    const int gk = gy * Kz + k;  // the column's Green entry at gx * Ky * Kz + gk
    const int KyKz = Ky * Kz;
    Cx<R>* la = a + cm.kk * ls;
    constexpr int U = 8;  // rows per round: their loads are issued together
    for (int x0 = cm.r0; x0 < Mx; x0 += U * cm.rs) {
        Cx<R> v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int x = x0 + u * cm.rs;
            v[u] = (x < nx && live) ? W[(size_t)x * ncol + col] : cx<R>(0, 0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (x0 + u * cm.rs < Mx) la[x0 + u * cm.rs] = v[u];
    }
    __syncthreads();
    Cx<R>* res = fft_lines<R, false, true, false>(a, b, ls, TK, rx, tw);
    Cx<R>* lr = res + cm.kk * ls;
    Cx<R>* lc = c + cm.kk * ls;
    for (int x0 = cm.r0; x0 < Mx; x0 += U * cm.rs) {
        R g[U];
        Cx<R> d[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int kx = x0 + u * cm.rs;
            const int gx = kx <= Mx - kx ? kx : Mx - kx;
            const long long gi = (long long)gx * KyKz + gk;
            g[u] = (kx < Mx && live && SC_IDX_OK(st, 23, gi, (long long)(rx.L / 2 + 1) * KyKz)) ? G[gi] : (R)0;
            d[u] = (W2 && kx < Mx) ? dx[kx] : cx<R>(0, 0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int kx = x0 + u * cm.rs;
            if (kx < Mx) {
                Cx<R> v = lr[kx];
                v.x *= g[u];
                v.y *= g[u];
                lr[kx] = v;
                if (W2) lc[kx] = cmul(v, d[u]);
            }
        }
    }
    __syncthreads();
    Cx<R>* res2 = fft_lines<R, true, true, false>(res, res == a ? b : a, ls, TK, rx, tw);
    if (live)
        for (int x = cm.r0; x < nx; x += cm.rs) W[(size_t)x * ncol + col] = res2[cm.kk * ls + x];
    if (W2) {
        __syncthreads();  // a and b are free
        Cx<R>* res3 = fft_lines<R, true, true, false>(c, a, ls, TK, rx, tw);
        if (live)
            for (int x = cm.r0; x < nx; x += cm.rs) W2[(size_t)x * ncol + col] = res3[cm.kk * ls + x];
    }
}

template <typename R>
__global__ void __launch_bounds__(FFT_THREADS<R>, FFT_MINB) k_xconv(Cx<R>* __restrict__ W, const R* __restrict__ G,
                                                       int nx, int My, int Kz, int Ky, RadixPlan rx,
                                                       const Cx<R>* __restrict__ twg, int TK, const ScState* st,
                                                       Spec<R> sp) {
    pdl_wait();
    xconv_body<R, ST_NO>(W, G, nx, My, Kz, Ky, rx, twg, TK, st, hw_vblk(), sp.W2, sp.dx);
}
template <int L>
__global__ void __launch_bounds__(stream_threads(L), stream_minb(L))
    k_xconv_s(Cx<float>* __restrict__ W, const float* __restrict__ G, int nx, int My, int Kz, int Ky, RadixPlan rx,
              const Cx<float>* __restrict__ twg, int TK, const ScState* st, Spec<float> sp) {
    pdl_wait();
    xconv_body<float, L>(W, G, nx, My, Kz, Ky, rx, twg, TK, st, hw_vblk(), sp.W2, sp.dx);
}

// Field outputs of the inverse passes (spectral fields, FP32): the grid a
// block writes, D(kz) applied before the z inverse or not, the factor 1/h of
// the difference and the plane left at zero (sc.py:196-198).
struct InvOut {
    int field;   // 0 potential, 1 Ex, 2 Ey, 3 Ez
    int nx;
};
template <typename R>
__device__ __forceinline__ void inv_out(const Spec<R>& sp, const ScState* st, int f, const Cx<R>* W, R* phi,
                                        const Cx<R>*& src, R*& out, const Cx<R>*& dz, R& mul) {
    src = f == 1 ? sp.W2 : (f == 2 && sp.W3 ? sp.W3 : W);
    out = f == 0 ? phi : (f == 1 ? sp.ex : (f == 2 ? sp.ey : sp.ez));
    dz = f == 3 ? sp.dz : nullptr;
    mul = f == 0 ? (R)1 : (R)st->istepsf[f - 1];
}

// dz != nullptr: the z spectrum is multiplied by D(kz) first; mul scales the
// output; zero_axis (0, 1, 2) leaves the last plane along that axis at zero
// (x = nx - 1, y = ny - 1 or z = nz - 1), -1 none
template <typename R>
__device__ __forceinline__ void zinv_body(const Cx<R>* __restrict__ W, R* __restrict__ phi, int ny, int nz, int My,
                                          int Kz, const RadixPlan& rz, const Cx<R>* __restrict__ twg, int NC,
                                          const ScState* st, VBlk vb, const Cx<R>* __restrict__ dz = nullptr,
                                          R mul = (R)1, int zero_axis = -1, int nx = 0) {
    extern __shared__ __align__(16) unsigned char smraw[];
    if (st->status) return;
    const int x = vb.y;
    const int y0 = vb.x * 2 * NC;
    OutScale64 out64 = {};
    if constexpr (sizeof(R) == 8) out64 = out_scale64(st);
    const R fscale = (R)st->phi_scalef * mul;  // (float)(norm / denom), computed once by the mesh finalize
    int pe = 0;  // FP64: the largest exponent stored
    auto put = [&](int c, int z, Cx<R> v) {
        if (z >= nz) return;
        const int ya = y0 + 2 * c, yb = ya + 1;
        if constexpr (sizeof(R) == 8) {
            double* p = phi + ((size_t)x * ny + ya) * nz + z;
            if (ya < ny) pe = max(pe, fx_exp(p[0] = out64(v.x)));
            if (yb < ny) pe = max(pe, fx_exp(p[nz] = out64(v.y)));
        } else {
            const bool zx = zero_axis == 0 && x == nx - 1, zz = zero_axis == 2 && z == nz - 1;
            const bool za = zx || zz || (zero_axis == 1 && ya == ny - 1);
            const bool zb = zx || zz || (zero_axis == 1 && yb == ny - 1);
            if (ya < ny) phi[((size_t)x * ny + ya) * nz + z] = za ? (R)0 : v.x * fscale;
            if (yb < ny) phi[((size_t)x * ny + yb) * nz + z] = zb ? (R)0 : v.y * fscale;
        }
    };
    const int Mz = rz.L, lz = fft_ls(Mz);
    Cx<R>* tw = reinterpret_cast<Cx<R>*>(smraw);
    Cx<R>* a = tw + Mz;
    Cx<R>* b = a + NC * lz;
    load_twiddles<R>(tw, twg, Mz);
    constexpr int U = 4;  // elements per thread per round, their loads issued together
    for (DivWalk w(threadIdx.x, blockDim.x, Mz); w.q < NC;) {
        int cs[U], ks[U];
        Cx<R> A[U], B[U], d[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            cs[u] = w.q;
            ks[u] = w.r;
            w.next();
            const int ya = y0 + 2 * cs[u], yb = ya + 1;
            const bool in = cs[u] < NC;
            const int kk = ks[u] < Kz ? ks[u] : Mz - ks[u];
            A[u] = (in && ya < ny) ? W[((size_t)x * My + ya) * Kz + kk] : cx<R>(0, 0);
            B[u] = (in && yb < ny) ? W[((size_t)x * My + yb) * Kz + kk] : cx<R>(0, 0);
            d[u] = (dz && in) ? dz[kk] : cx<R>(0, 0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (cs[u] >= NC) continue;
            Cx<R> Au = A[u], Bu = B[u];
            if (dz) {
                Au = cmul(Au, d[u]);
                Bu = cmul(Bu, d[u]);
            }
            // Z = A + iB, Hermitian-extended above Mz/2
            a[cs[u] * lz + ks[u]] = ks[u] < Kz ? cx<R>(Au.x - Bu.y, Au.y + Bu.x) : cx<R>(Au.x + Bu.y, Bu.x - Au.y);
        }
    }
    __syncthreads();
    Cx<R>* res = fft_lines<R, true, true, sizeof(R) == 4>(a, b, lz, NC, rz, tw);
    for (DivWalk w(threadIdx.x, blockDim.x, nz); w.q < NC; w.next()) put(w.q, w.r, res[w.q * lz + w.r]);
    if constexpr (sizeof(R) == 8) phi_raise(st, pe);
}

// blockIdx.z: the output (0 the potential; with spectral fields 1 Ex, 2 Ey, 3 Ez)
template <typename R>
__global__ void __launch_bounds__(FFT_THREADS<R>, FFT_MINB) k_zinv(const Cx<R>* __restrict__ W, R* __restrict__ phi,
                                                      int ny, int nz, int My, int Kz, RadixPlan rz,
                                                      const Cx<R>* __restrict__ twg, int NC,
                                                      const ScState* st, Spec<R> sp) {
    pdl_wait();
    const int f = (int)blockIdx.z + sp.f0;
    const Cx<R>* src;
    R* out;
    const Cx<R>* dz;
    R mul;
    inv_out<R>(sp, st, f, W, phi, src, out, dz, mul);
    zinv_body<R>(src, out, ny, nz, My, Kz, rz, twg, NC, st, hw_vblk(), dz, mul, f - 1, (int)gridDim.y);
}

template <int L>
__global__ void __launch_bounds__(fx_threads(L), FX_MINB(L)) k_zinv_fx(const double2* __restrict__ W,
                                                                    double* __restrict__ phi, int ny, int nz, int My,
                                                                    int Kz, const double2* __restrict__ twg, int NC,
                                                                    const ScState* st) {
    pdl_wait();
    if (st->status) return;
    zinv_fx<L>(W, phi, ny, nz, My, Kz, twg, NC, out_scale64(st), st, hw_vblk());
}

// FP64 form: Ex,Ey,Ez = forward differences / h, zero on the last plane
// (sc.py:195-200); the quotient from the reciprocal 1/h with one correction
// (the IEEE division's result up to its last bit).  One block per (x, y) line
// of cells, one thread per z: no index division.
//
// fe != nullptr (the kick): the differences also as integers under the
// potential's largest exponent, [3][nx][ny][nz]; differences of integers are
// exact, and an integer's unit is 2^-59 of the largest potential, a 64th of
// what the double potential itself is rounded at.  escale turns them into fields.
__global__ void k_field_grids(const double* __restrict__ phi, double* __restrict__ ex, double* __restrict__ ey,
                              double* __restrict__ ez, long long* __restrict__ fe, int nx, int ny, int nz,
                              ScState* st) {
    pdl_wait();
    if (st->status) return;
    const int j = blockIdx.x, i = blockIdx.y;
    const double hx = st->steps[0], hy = st->steps[1], hz = st->steps[2];
    const double rx = st->isteps[0], ry = st->isteps[1], rz = st->isteps[2];
    const int E = max(st->phi_exp, 1);  // denormals have exponent 1
    const size_t ncell = (size_t)nx * ny * nz;
    if (fe && i == 0 && j == 0 && threadIdx.x < 3) {
        const int a = threadIdx.x;
        const double sc = E == FX_BAD ? NAN : ldexp(st->isteps[a], E - 1023);
        st->escale[a] = sc;
        for (int b = 0; b < 3; ++b)
            st->Tke[b][a] = E == FX_BAD ? NAN : ldexp(st->Tk[b][a] * st->isteps[a], E - 1023);
    }
    auto over = [](double a, double h, double r) {
        const double q = a * r;
        return fma(fma(-q, h, a), r, q);
    };
    for (int k = threadIdx.x; k < nz; k += blockDim.x) {
        const int c = (i * ny + j) * nz + k;
        const bool inx = i < nx - 1, iny = j < ny - 1, inz = k < nz - 1;
        const double p = phi[c];
        const double px = inx ? phi[c + ny * nz] : p, py = iny ? phi[c + nz] : p, pz = inz ? phi[c + 1] : p;
        ex[c] = inx ? over(p - px, hx, rx) : 0.0;
        ey[c] = iny ? over(p - py, hy, ry) : 0.0;
        ez[c] = inz ? over(p - pz, hz, rz) : 0.0;
        if (fe) {
            const Fx f = fx_from<FX_PHI>(p, E);
            fe[c] = (f - fx_from<FX_PHI>(px, E)).v;
            fe[ncell + c] = (f - fx_from<FX_PHI>(py, E)).v;
            fe[2 * ncell + c] = (f - fx_from<FX_PHI>(pz, E)).v;
        }
    }
}

// FP32 form: the field grids as "octs" for the gather -- for each cell
// (i,j,k) and each component F, the 8 values F[i+a][j+b][k+c] (a, b, c in
// {0,1}) at index 4a + 2b + c, 32 bytes aligned to 32; a trilinear sample
// then reads one 32-byte sector instead of eight scalars.  Entries that the
// gather never uses (i = nx-1, j = ny-1 or k = nz-1 as a base) are written
// but not read.
__device__ __forceinline__ float fd(const float* __restrict__ phi, int i, int j, int k, int di, int dj, int dk,
                                    int nx, int ny, int nz, float ih) {
    // forward difference along (di,dj,dk), zero on the last plane and outside the grid
    if (i >= nx || j >= ny || k >= nz) return 0.f;
    if (i + di >= nx || j + dj >= ny || k + dk >= nz) return 0.f;
    const int c = (i * ny + j) * nz + k;
    return (phi[c] - phi[c + (di * ny + dj) * nz + dk]) * ih;
}

__device__ __forceinline__ void st_oct(float* p, const float (&o)[8]) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(o[0]), "f"(o[1]), "f"(o[2]),
                 "f"(o[3]), "f"(o[4]), "f"(o[5]), "f"(o[6]), "f"(o[7])
                 : "memory");
}

__device__ __forceinline__ void field_octs_body(const float* __restrict__ phi, float* __restrict__ ox,
                                                float* __restrict__ oy, float* __restrict__ oz, int nx, int ny,
                                                int nz, const ScState* st, VBlk vb) {
    if (st->status) return;
    const int j = vb.x, i = vb.y;
    const float ih[3] = {st->istepsf[0], st->istepsf[1], st->istepsf[2]};
    float* const out[3] = {ox, oy, oz};
    for (int k = threadIdx.x; k < nz; k += blockDim.x) {
        const size_t c = ((size_t)i * ny + j) * nz + k;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            float o[8];
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < 2; ++b)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        o[4 * a + 2 * b + e] = fd(phi, i + a, j + b, k + e, d == 0, d == 1, d == 2, nx, ny, nz, ih[d]);
            st_oct(out[d] + 8 * c, o);
        }
    }
}

__global__ void k_field_octs(const float* __restrict__ phi, float* __restrict__ ox, float* __restrict__ oy,
                             float* __restrict__ oz, int nx, int ny, int nz, const ScState* st) {
    pdl_wait();
    field_octs_body(phi, ox, oy, oz, nx, ny, nz, st, hw_vblk());
}

// the octs of field grids computed in Fourier space (spectral fields): the 8
// neighbouring values themselves, zero outside the grid
__device__ __forceinline__ float at_or0(const float* __restrict__ F, int i, int j, int k, int nx, int ny, int nz) {
    return (i < nx && j < ny && k < nz) ? F[((size_t)i * ny + j) * nz + k] : 0.f;
}
__device__ __forceinline__ void field_octs_spectral_body(const float* __restrict__ ex, const float* __restrict__ ey,
                                                         const float* __restrict__ ez, float* __restrict__ ox,
                                                         float* __restrict__ oy, float* __restrict__ oz, int nx,
                                                         int ny, int nz, const ScState* st, VBlk vb) {
    if (st->status) return;
    const int j = vb.x, i = vb.y;
    const float* const in[3] = {ex, ey, ez};
    float* const out[3] = {ox, oy, oz};
    for (int k = threadIdx.x; k < nz; k += blockDim.x) {
        const size_t c = ((size_t)i * ny + j) * nz + k;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            float o[8];
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < 2; ++b)
#pragma unroll
                    for (int e = 0; e < 2; ++e) o[4 * a + 2 * b + e] = at_or0(in[d], i + a, j + b, k + e, nx, ny, nz);
            st_oct(out[d] + 8 * c, o);
        }
    }
}
__global__ void k_field_octs_spectral(const float* __restrict__ ex, const float* __restrict__ ey,
                                      const float* __restrict__ ez, float* __restrict__ ox, float* __restrict__ oy,
                                      float* __restrict__ oz, int nx, int ny, int nz, const ScState* st) {
    pdl_wait();
    field_octs_spectral_body(ex, ey, ez, ox, oy, oz, nx, ny, nz, st, hw_vblk());
}


// ---------------------------------------------------------------------------
// Plane-fused passes (meshes whose y-by-kz plane fits in shared memory): one
// block per x plane does the z and y forward transforms (F1 + F2), or the y
// and z inverse transforms (B2 + B1), keeping the plane in shared memory
// between them.  The lines go through the same fft_lines code as the
// separate passes, so the results are identical; the plane saves a kernel
// launch and a round trip of the work grid per direction.
// Shared memory: twiddles z and y, then two buffers of Kz y-lines; the z
// lines use the second buffer (forward) or whichever buffer the y result
// does not occupy (inverse).
// ---------------------------------------------------------------------------
// FP64: 512, for the 128 registers of the fixed-point transforms
template <typename R>
constexpr int PLANE_THREADS = sizeof(R) == 8 ? 512 : 1024;

template <typename R>
static size_t plane_smem(const Plan& p) {
    const int Kz = p.Mz / 2 + 1;
    return sizeof(Cx<R>) * ((size_t)p.Mz + p.My + 2 * (size_t)Kz * fft_ls(p.My));
}
template <typename R>
static bool plane_fits(const Plan& p, int optin) {
    const int Kz = p.Mz / 2 + 1, ncz = (p.ny + 1) / 2;
    return 2 * (size_t)ncz * fft_ls(p.Mz) <= (size_t)Kz * fft_ls(p.My) && plane_smem<R>(p) <= (size_t)optin;
}

template <typename R>
__device__ __forceinline__ void zy_fwd_body(R* __restrict__ q, const long long* __restrict__ qfix,
                                            Cx<R>* __restrict__ W, int ny, int nz, int My, int Kz,
                                            const RadixPlan& rz, const RadixPlan& ry, const Cx<R>* __restrict__ twzg,
                                            const Cx<R>* __restrict__ twyg, const ScState* st, int x, int nx) {
    extern __shared__ __align__(16) unsigned char smraw[];
    if (st->status) return;
    const int Mz = rz.L, lz = fft_ls(Mz), ly = fft_ls(My), ncz = (ny + 1) / 2;
    Cx<R>* twz = reinterpret_cast<Cx<R>*>(smraw);
    Cx<R>* twy = twz + Mz;
    Cx<R>* A2 = twy + My;
    Cx<R>* B2 = A2 + Kz * ly;
    Cx<R>* A1 = B2;
    Cx<R>* B1 = A1 + ncz * lz;
    load_twiddles<R>(twz, twzg, Mz);
    load_twiddles<R>(twy, twyg, My);
    // F1: two charge rows per complex line (as k_zfwd)
    stage_charge_lines<R>(q, qfix, A1, lz, x, 0, ncz, ny, nz, Mz, st, (long long)nx * ny * nz, 25);
    __syncthreads();
    const Cx<R>* res1 = fft_lines<R, false, true>(A1, B1, lz, ncz, rz, twz);
    // unpack the two real lines into the y lines (column kz, row y); rows
    // ny..My-1 are the zero padding of F2
    for (DivWalk w(threadIdx.x, blockDim.x, Kz); w.q < ncz; w.next()) {
        const int c = w.q, k = w.r;
        const int ya = 2 * c, yb = ya + 1;
        const Cx<R> Z = res1[c * lz + k];
        const Cx<R> Zm = res1[c * lz + (k == 0 ? 0 : Mz - k)];
        const R h = unpack_half<R>();
        A2[k * ly + ya] = scaled<R>(Z.x + Zm.x, Z.y - Zm.y, h);
        if (yb < ny) A2[k * ly + yb] = scaled<R>(Z.y + Zm.y, Zm.x - Z.x, h);
    }
    for (DivWalk w(threadIdx.x, blockDim.x, Kz); w.q < My - ny; w.next()) A2[w.r * ly + ny + w.q] = cx<R>(0, 0);
    __syncthreads();
    const Cx<R>* res2 = fft_lines<R, false, true>(A2, B2, ly, Kz, ry, twy);
    Cx<R>* Wx = W + (size_t)x * My * Kz;  // the plane: row ky, column k at ky * Kz + k
    for (DivWalk w(threadIdx.x, blockDim.x, Kz); w.q < My; w.next()) Wx[w.q * Kz + w.r] = res2[w.r * ly + w.q];
}

template <typename R>
__global__ void __launch_bounds__(PLANE_THREADS<R>) k_zy_fwd(R* __restrict__ q, const long long* __restrict__ qfix,
                                                          Cx<R>* __restrict__ W, int ny, int nz, int My, int Kz,
                                                          RadixPlan rz, RadixPlan ry, const Cx<R>* __restrict__ twz,
                                                          const Cx<R>* __restrict__ twy, const ScState* st) {
    pdl_wait();
    zy_fwd_body<R>(q, qfix, W, ny, nz, My, Kz, rz, ry, twz, twy, st, (int)blockIdx.x, (int)gridDim.x);
}

// dy / dz != nullptr (spectral fields): the plane is multiplied by D(ky)
// before the y inverse / by D(kz) before the z inverse; mul and zero_axis as
// in zinv_body
template <typename R>
__device__ __forceinline__ void yz_inv_body(const Cx<R>* __restrict__ W, R* __restrict__ phi, int ny, int nz,
                                            int My, int Kz, const RadixPlan& rz, const RadixPlan& ry,
                                            const Cx<R>* __restrict__ twzg, const Cx<R>* __restrict__ twyg,
                                            const ScState* st, int x, const Cx<R>* __restrict__ dy = nullptr,
                                            const Cx<R>* __restrict__ dz = nullptr, R mul = (R)1,
                                            int zero_axis = -1, int nx = 0) {
    extern __shared__ __align__(16) unsigned char smraw[];
    if (st->status) return;
    const int Mz = rz.L, lz = fft_ls(Mz), ly = fft_ls(My), ncz = (ny + 1) / 2;
    Cx<R>* twz = reinterpret_cast<Cx<R>*>(smraw);
    Cx<R>* twy = twz + Mz;
    Cx<R>* A2 = twy + My;
    Cx<R>* B2 = A2 + Kz * ly;
    load_twiddles<R>(twz, twzg, Mz);
    load_twiddles<R>(twy, twyg, My);
    const Cx<R>* Wx = W + (size_t)x * My * Kz;
    constexpr int U = 4;  // elements per thread per round, their loads issued together
    for (DivWalk w(threadIdx.x, blockDim.x, Kz); w.q < My;) {
        int ys[U], ks[U];
        Cx<R> v[U], d[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            ys[u] = w.q;
            ks[u] = w.r;
            w.next();
            const bool in = ys[u] < My;
            v[u] = in ? Wx[ys[u] * Kz + ks[u]] : cx<R>(0, 0);
            d[u] = (dy && in) ? dy[ys[u]] : cx<R>(0, 0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (ys[u] < My) A2[ks[u] * ly + ys[u]] = dy ? cmul(v[u], d[u]) : v[u];
    }
    __syncthreads();
    // B2: inverse y; only rows y < ny are used
    const Cx<R>* res2 = fft_lines<R, true, true>(A2, B2, ly, Kz, ry, twy);
    Cx<R>* A1 = res2 == B2 ? A2 : B2;
    Cx<R>* B1 = A1 + ncz * lz;
    // B1: two output rows per complex line, Hermitian-extended (as k_zinv)
    for (DivWalk w(threadIdx.x, blockDim.x, Mz); w.q < ncz; w.next()) {
        const int c = w.q, k = w.r;
        const int ya = 2 * c, yb = ya + 1;
        const bool lo = k < Kz;
        const int kk = lo ? k : Mz - k;
        Cx<R> A = res2[kk * ly + ya];
        Cx<R> B = yb < ny ? res2[kk * ly + yb] : cx<R>(0, 0);
        if (dz) {
            A = cmul(A, dz[kk]);
            B = cmul(B, dz[kk]);
        }
        A1[c * lz + k] = lo ? cx<R>(A.x - B.y, A.y + B.x) : cx<R>(A.x + B.y, B.x - A.y);
    }
    __syncthreads();
    const Cx<R>* res = fft_lines<R, true, true>(A1, B1, lz, ncz, rz, twz);
    OutScale64 out64 = {};
    if constexpr (sizeof(R) == 8) out64 = out_scale64(st);
    const R fscale = (R)st->phi_scalef * mul;  // (float)(norm / denom), computed once by the mesh finalize
    int pe = 0;  // FP64: the largest exponent stored
    for (DivWalk w(threadIdx.x, blockDim.x, nz); w.q < ncz; w.next()) {
        const int c = w.q, z = w.r;
        const int ya = 2 * c, yb = ya + 1;
        const Cx<R> v = res[c * lz + z];
        if constexpr (sizeof(R) == 8) {
            double* p = phi + ((size_t)x * ny + ya) * nz + z;
            pe = max(pe, fx_exp(p[0] = out64(v.x)));
            if (yb < ny) pe = max(pe, fx_exp(p[nz] = out64(v.y)));
        } else {
            const bool zx = zero_axis == 0 && x == nx - 1, zz = zero_axis == 2 && z == nz - 1;
            const bool za = zx || zz || (zero_axis == 1 && ya == ny - 1);
            const bool zb = zx || zz || (zero_axis == 1 && yb == ny - 1);
            phi[((size_t)x * ny + ya) * nz + z] = za ? (R)0 : v.x * fscale;
            if (yb < ny) phi[((size_t)x * ny + yb) * nz + z] = zb ? (R)0 : v.y * fscale;
        }
    }
    if constexpr (sizeof(R) == 8) phi_raise(st, pe);
}

// blockIdx.y: the output (0 the potential; with spectral fields 1 Ex, 2 Ey, 3 Ez)
template <typename R>
__global__ void __launch_bounds__(PLANE_THREADS<R>) k_yz_inv(const Cx<R>* __restrict__ W, R* __restrict__ phi, int ny,
                                                          int nz, int My, int Kz, RadixPlan rz, RadixPlan ry,
                                                          const Cx<R>* __restrict__ twz,
                                                          const Cx<R>* __restrict__ twy, const ScState* st,
                                                          Spec<R> sp) {
    pdl_wait();
    const int f = (int)blockIdx.y + sp.f0;
    const Cx<R>* src;
    R* out;
    const Cx<R>* dz;
    R mul;
    Spec<R> spp = sp;
    spp.W3 = nullptr;  // the plane pass applies D(ky) itself
    inv_out<R>(spp, st, f, W, phi, src, out, dz, mul);
    yz_inv_body<R>(src, out, ny, nz, My, Kz, rz, ry, twz, twy, st, (int)blockIdx.x, f == 2 ? sp.dy : nullptr, dz,
                   mul, f - 1, (int)gridDim.x);
}

static int optin_smem();
// the plane-fused passes are used where the plane fits shared memory and the
// plan's parameters (SC_PARAM_FFT_PLANE_FWD / _INV) allow them
static bool plane_ok(const Plan& p) {
    return p.prec == SC_FP64 ? plane_fits<double>(p, optin_smem()) : plane_fits<float>(p, optin_smem());
}
int convolve_launches(const Plan& p) {
    const bool plane = plane_ok(p);
    return (plane && p.fft_plane_fwd ? 1 : 2) + 1 + (plane && p.fft_plane_inv ? 1 : 2);
}

static int optin_smem() {
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) || cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) return 0;
    return v;
}

// the spectral-field pointers of a plan's workspace (W2 == nullptr: none)
// want_phi: the inverse passes also produce the potential (the kick's field
// octs do not read it; an inspection or the record-field mode does)
template <typename R>
__host__ __device__ __forceinline__ Spec<R> spec_of(const Plan& p, const Layout& L, char* ws, bool fields,
                                                    bool want_phi = true) {
    Spec<R> sp = {};
    if (!(fields && p.spectral && sizeof(R) == 4)) return sp;
    sp.f0 = want_phi ? 0 : 1;
    sp.W2 = reinterpret_cast<Cx<R>*>(ws + L.W2);
    sp.W3 = reinterpret_cast<Cx<R>*>(ws + L.W3);
    sp.dx = reinterpret_cast<const Cx<R>*>(ws + L.dt_x);
    sp.dy = reinterpret_cast<const Cx<R>*>(ws + L.dt_y);
    sp.dz = reinterpret_cast<const Cx<R>*>(ws + L.dt_z);
    sp.ex = reinterpret_cast<R*>(ws + L.ex);
    sp.ey = reinterpret_cast<R*>(ws + L.ey);
    sp.ez = reinterpret_cast<R*>(ws + L.ez);
    return sp;
}

// Launches of the separate passes: the kernel of the line length (FP32
// streamed, FP64 fixed point) for the two-step lengths, the staged one for others.
template <typename R>
static cudaError_t launch_zfwd(const Plan& p, dim3 g, size_t sm, cudaStream_t s, R* q, const long long* qfix, Cx<R>* W,
                               int Kz, const Cx<R>* tw, int NC, const ScState* st) {
    cudaError_t e;
    if (uses_two_step(p.Mz))
        return two_step_host(p.Mz, [&](auto L) -> cudaError_t {
            constexpr int LL = decltype(L)::value;
            if constexpr (sizeof(R) == 4) {
                if ((e = set_smem(k_zfwd_s<LL>, sm))) return e;
                return launch(k_zfwd_s<LL>, g, 128, sm, s, q, qfix, W, p.ny, p.nz, p.My, Kz, p.rz, tw, NC, st);
            } else {
                if ((e = set_smem(k_zfwd_fx<LL>, sm))) return e;
                return launch(k_zfwd_fx<LL>, g, NC * two_step_q(LL), sm, s, q, W, p.ny, p.nz, p.My, Kz, tw, NC, st);
            }
        });
    if ((e = set_smem(k_zfwd<R>, sm))) return e;
    return launch(k_zfwd<R>, g, FFT_THREADS<R>, sm, s, q, qfix, W, p.ny, p.nz, p.My, Kz, p.rz, tw, NC, st);
}
template <typename R, bool INV>
static cudaError_t launch_ypass(const Plan& p, dim3 g, size_t sm, cudaStream_t s, Cx<R>* W, int Kz, const Cx<R>* tw,
                                int TK, const ScState* st, const Spec<R>& sp) {
    cudaError_t e;
    if (uses_two_step(p.My))
        return two_step_host(p.My, [&](auto L) -> cudaError_t {
            constexpr int LL = decltype(L)::value;
            if constexpr (sizeof(R) == 4) {
                if ((e = set_smem(k_ypass_s<INV, LL>, sm))) return e;
                return launch(k_ypass_s<INV, LL>, g, stream_threads(LL), sm, s, W, p.nx, p.ny, p.My, Kz, p.ry, tw, TK, st,
                              sp);
            } else {
                if ((e = set_smem(k_ypass_fx<INV, LL>, sm))) return e;
                return launch(k_ypass_fx<INV, LL>, g, fx_threads_xy(LL), sm, s, W, p.nx, p.ny, Kz, tw, st);
            }
        });
    if ((e = set_smem(k_ypass<R, INV>, sm))) return e;
    return launch(k_ypass<R, INV>, g, FFT_THREADS<R>, sm, s, W, p.nx, p.ny, p.My, Kz, p.ry, tw, TK, st, sp);
}
template <typename R>
static cudaError_t launch_xconv(const Plan& p, dim3 g, size_t sm, cudaStream_t s, Cx<R>* W, const R* G, int Kz, int Ky,
                                const Cx<R>* tw, int TK, const ScState* st, const Spec<R>& sp) {
    cudaError_t e;
    if (uses_two_step(p.Mx))
        return two_step_host(p.Mx, [&](auto L) -> cudaError_t {
            constexpr int LL = decltype(L)::value;
            if constexpr (sizeof(R) == 4) {
                if ((e = set_smem(k_xconv_s<LL>, sm))) return e;
                return launch(k_xconv_s<LL>, g, stream_threads(LL), sm, s, W, G, p.nx, p.My, Kz, Ky, p.rx, tw, TK, st, sp);
            } else {
                if ((e = set_smem(k_xconv_fx<LL>, sm))) return e;
                return launch(k_xconv_fx<LL>, g, fx_threads_xy(LL), sm, s, W, G, p.nx, p.My, Kz, Ky, tw, st);
            }
        });
    if ((e = set_smem(k_xconv<R>, sm))) return e;
    return launch(k_xconv<R>, g, FFT_THREADS<R>, sm, s, W, G, p.nx, p.My, Kz, Ky, p.rx, tw, TK, st, sp);
}

template <typename R>
static cudaError_t convolve_t(const Plan& p, const Layout& L, char* ws, R* qgrid, R* phi, const long long* qfix,
                              cudaStream_t s, int part, bool fields, bool want_phi) {
    const ScState* st = reinterpret_cast<const ScState*>(ws + L.state);
    const int Kz = p.Mz / 2 + 1, Ky = p.My / 2 + 1;
    const Spec<R> sp = spec_of<R>(p, L, ws, fields, want_phi);
    const int nbuf = sp.W2 ? 3 : 2;  // line buffers of the x pass and the y inverse
    Cx<R>* W = reinterpret_cast<Cx<R>*>(ws + L.W);
    const R* G = reinterpret_cast<const R*>(ws + L.green);
    const Cx<R>* twx = reinterpret_cast<const Cx<R>*>(ws + L.tw_x);
    const Cx<R>* twy = reinterpret_cast<const Cx<R>*>(ws + L.tw_y);
    const Cx<R>* twz = reinterpret_cast<const Cx<R>*>(ws + L.tw_z);
    cudaError_t e;
    const int NC = z_lines<R>(p.Mz);
    const size_t smz = smem_zf<R>(p.Mz, NC), smzi = smem_zi<R>(p.Mz, NC);
    dim3 gz((p.ny + 2 * NC - 1) / (2 * NC), p.nx);
    const int tky = pass_cols<R>(p.fft_cols_y, p.My), tkx = pass_cols<R>(p.fft_cols_x, p.Mx, nbuf);
    const int tkyi = pass_cols<R>(p.fft_cols_y, p.My, nbuf);  // the y inverse
    const size_t smy = smem_yf<R>(p.My, tky), smyi = smem_yi<R>(p.My, tkyi, sp.W2 != nullptr);
    const int ycols = p.nx * Kz;  // the y passes' columns (x, kz)
    dim3 gy((ycols + tky - 1) / tky);
    dim3 gyi((ycols + tkyi - 1) / tkyi, sp.W2 ? 2 : 1);
    static const int optin = optin_smem();
    const bool plane = plane_fits<R>(p, optin);
    const bool plane_fwd = plane && p.fft_plane_fwd, plane_inv = plane && p.fft_plane_inv;
    const size_t smp = plane_smem<R>(p);
    if (plane_fwd && part != CONV_REST) {
        if ((e = set_smem(k_zy_fwd<R>, smp))) return e;
        launch(k_zy_fwd<R>, p.nx, PLANE_THREADS<R>, smp, s, qgrid, qfix, W, p.ny, p.nz, p.My, Kz, p.rz, p.ry, twz, twy, st);
    } else if (part != CONV_REST) {
        if ((e = launch_zfwd<R>(p, gz, smz, s, qgrid, qfix, W, Kz, twz, NC, st))) return e;
        if ((e = launch_ypass<R, false>(p, gy, smy, s, W, Kz, twy, tky, st, Spec<R>{}))) return e;
    }
    if (part == CONV_FORWARD) return cudaGetLastError();
    const size_t smx = smem_x<R>(p.Mx, tkx, sp.W2 != nullptr);
    dim3 gx((p.My * Kz + tkx - 1) / tkx);  // the x pass's columns (ky, kz)
    if ((e = launch_xconv<R>(p, gx, smx, s, W, G, Kz, Ky, twx, tkx, st, sp))) return e;
    const int nout = sp.W2 ? 4 - sp.f0 : 1;  // [the potential,] Ex, Ey, Ez
    if (plane_inv) {
        if ((e = set_smem(k_yz_inv<R>, smp))) return e;
        launch(k_yz_inv<R>, dim3(p.nx, nout), PLANE_THREADS<R>, smp, s, W, phi, p.ny, p.nz, p.My, Kz, p.rz, p.ry, twz, twy,
               st, sp);
        return cudaGetLastError();
    }
    if ((e = launch_ypass<R, true>(p, gyi, smyi, s, W, Kz, twy, tkyi, st, sp))) return e;
    if (sizeof(R) == 8 && uses_two_step(p.Mz)) {
        if constexpr (sizeof(R) == 8)
            return two_step_host(p.Mz, [&](auto LZ) -> cudaError_t {
                constexpr int LL = decltype(LZ)::value;
                if ((e = set_smem(k_zinv_fx<LL>, smzi))) return e;
                return launch(k_zinv_fx<LL>, gz, NC * two_step_q(LL), smzi, s, W, phi, p.ny, p.nz, p.My, Kz, twz, NC, st);
            });
    }
    if ((e = set_smem(k_zinv<R>, smzi))) return e;
    launch(k_zinv<R>, dim3(gz.x, gz.y, nout), FFT_THREADS<R>, smzi, s, W, phi, p.ny, p.nz, p.My, Kz, p.rz, twz, NC, st, sp);
    return cudaGetLastError();
}

template <typename R>
static cudaError_t prepare_fft_t(const Plan& p) {
    cudaError_t e;
    const int NC = z_lines<R>(p.Mz);
    const size_t smz = smem_zf<R>(p.Mz, NC), smzi = smem_zi<R>(p.Mz, NC);
    const bool spec = p.spectral && sizeof(R) == 4;
    const int nbuf = spec ? 3 : 2;
    const int tky = strided_cols<R>(p.My), tkx = strided_cols<R>(p.Mx, nbuf), tkyi = strided_cols<R>(p.My, nbuf);
    const size_t smy = smem_yf<R>(p.My, tky), smyi = smem_yi<R>(p.My, tkyi, spec), smx = smem_x<R>(p.Mx, tkx, spec);
    auto prep = [&](int M, auto&& two_step, auto* staged, size_t sm) -> cudaError_t {
        return uses_two_step(M) ? two_step_host(M, two_step) : set_smem(staged, sm);
    };
    if ((e = prep(p.Mz, [&](auto L) {
             constexpr int LL = decltype(L)::value;
             if constexpr (sizeof(R) == 4) return set_smem(k_zfwd_s<LL>, smz);
             else return set_smem(k_zfwd_fx<LL>, smz);
         }, k_zfwd<R>, smz))) return e;
    if ((e = prep(p.My, [&](auto L) {
             constexpr int LL = decltype(L)::value;
             if constexpr (sizeof(R) == 4) return set_smem(k_ypass_s<false, LL>, smy);
             else return set_smem(k_ypass_fx<false, LL>, smy);
         }, k_ypass<R, false>, smy))) return e;
    if ((e = prep(p.My, [&](auto L) {
             constexpr int LL = decltype(L)::value;
             if constexpr (sizeof(R) == 4) return set_smem(k_ypass_s<true, LL>, smyi);
             else return set_smem(k_ypass_fx<true, LL>, smyi);
         }, k_ypass<R, true>, smyi))) return e;
    if ((e = prep(p.Mx, [&](auto L) {
             constexpr int LL = decltype(L)::value;
             if constexpr (sizeof(R) == 4) return set_smem(k_xconv_s<LL>, smx);
             else return set_smem(k_xconv_fx<LL>, smx);
         }, k_xconv<R>, smx))) return e;
    if ((e = prep(p.Mz, [&](auto L) {
             if constexpr (sizeof(R) == 4) return set_smem(k_zinv<R>, smzi);
             else return set_smem(k_zinv_fx<decltype(L)::value>, smzi);
         }, k_zinv<R>, smzi))) return e;
    if (plane_fits<R>(p, optin_smem())) {
        if ((e = set_smem(k_zy_fwd<R>, plane_smem<R>(p)))) return e;
        if ((e = set_smem(k_yz_inv<R>, plane_smem<R>(p)))) return e;
    }
    return cudaSuccess;
}

cudaError_t prepare_fft_kernels(const Plan& p) {
    return p.prec == SC_FP64 ? prepare_fft_t<double>(p) : prepare_fft_t<float>(p);
}

cudaError_t launch_convolve(const Plan& p, const Layout& L, char* ws, const void* qgrid_in, void* phi_out,
                            cudaStream_t s, const long long* qfix, int part, bool fields, bool want_phi) {
    if (p.prec == SC_FP64)
        return convolve_t<double>(p, L, ws, static_cast<double*>(const_cast<void*>(qgrid_in)),
                                  static_cast<double*>(phi_out), nullptr, s, part, false, true);
    return convolve_t<float>(p, L, ws, static_cast<float*>(const_cast<void*>(qgrid_in)), static_cast<float*>(phi_out),
                             qfix, s, part, fields, want_phi);
}

template <typename R>
static cudaError_t field_t(const Plan& p, const Layout& L, char* ws, cudaStream_t s, bool kick) {
    const ScState* st = reinterpret_cast<const ScState*>(ws + L.state);
    const int bt = p.nz < 256 ? ((p.nz + 31) / 32) * 32 : 256;
    const dim3 grid(p.ny, p.nx);
    if (sizeof(R) == 4 && p.spectral)
        launch(k_field_octs_spectral, grid, bt, 0, s, reinterpret_cast<const float*>(ws + L.ex),
               reinterpret_cast<const float*>(ws + L.ey), reinterpret_cast<const float*>(ws + L.ez),
               reinterpret_cast<float*>(ws + L.exq), reinterpret_cast<float*>(ws + L.eyq),
               reinterpret_cast<float*>(ws + L.ezq), p.nx, p.ny, p.nz, st);
    else if (sizeof(R) == 4)
        launch(k_field_octs, grid, bt, 0, s, reinterpret_cast<const float*>(ws + L.phi), reinterpret_cast<float*>(ws + L.exq),
                                         reinterpret_cast<float*>(ws + L.eyq), reinterpret_cast<float*>(ws + L.ezq),
                                         p.nx, p.ny, p.nz, st);
    else
        launch(k_field_grids, grid, bt, 0, s, reinterpret_cast<const double*>(ws + L.phi),
               reinterpret_cast<double*>(ws + L.ex), reinterpret_cast<double*>(ws + L.ey),
               reinterpret_cast<double*>(ws + L.ez), kick ? field_fx(L, ws) : nullptr, p.nx, p.ny, p.nz,
               reinterpret_cast<ScState*>(ws + L.state));
    return cudaGetLastError();
}

cudaError_t launch_field_grids(const Plan& p, const Layout& L, char* ws, cudaStream_t s, bool kick) {
    return p.prec == SC_FP64 ? field_t<double>(p, L, ws, s, kick) : field_t<float>(p, L, ws, s, kick);
}

// ---------------------------------------------------------------------------
// batched convolution and field (FP32 form): one launch per pass over every
// beam of a batch, each beam with the tiling of its plain launch
// ---------------------------------------------------------------------------
#define BATCH_BEAM(stage)                                                       \
    const int b = batch_beam(start, nb);                                        \
    const BatchBeam& B = beams[b];                                              \
    const VBlk vb = batch_vblk(start, b, B.gx[stage], B.gy[stage]);             \
    char* ws = B.ws;                                                            \
    const Layout& L = B.L;                                                      \
    const Plan& p = B.p;                                                        \
    const ScState* st = reinterpret_cast<const ScState*>(ws + L.state);

__global__ void __launch_bounds__(FFT_THREADS<float>, FFT_MINB) kb_zfwd(const BatchBeam* __restrict__ beams,
                                                       const int* __restrict__ start, int nb) {
    pdl_wait();
    BATCH_BEAM(BS_FFT_Z)
    zfwd_body<float, ST_ANY>(reinterpret_cast<float*>(ws + L.qgrid), reinterpret_cast<const long long*>(ws + L.qfix),
                     reinterpret_cast<Cx<float>*>(ws + L.W), p.ny, p.nz, p.My, p.Mz / 2 + 1, p.rz,
                     reinterpret_cast<const Cx<float>*>(ws + L.tw_z), B.fft_nc, st, vb);
}

// forward y pass
__global__ void __launch_bounds__(FFT_THREADS<float>, FFT_MINB) kb_yfwd(const BatchBeam* __restrict__ beams,
                                                       const int* __restrict__ start, int nb) {
    pdl_wait();
    BATCH_BEAM(BS_FFT_Y)
    ypass_body<float, false, ST_ANY>(reinterpret_cast<Cx<float>*>(ws + L.W), p.nx, p.ny, p.My, p.Mz / 2 + 1, p.ry,
                             reinterpret_cast<const Cx<float>*>(ws + L.tw_y), B.fft_tky, st, vb);
}

// inverse y pass: block row 0 takes W (and, with spectral fields, W x D(ky)
// into W3), row 1 the x-differenced W2 (as k_ypass's blockIdx.y)
__global__ void __launch_bounds__(FFT_THREADS<float>, FFT_MINB) kb_yinv(const BatchBeam* __restrict__ beams,
                                                       const int* __restrict__ start, int nb) {
    pdl_wait();
    BATCH_BEAM(BS_FFT_YI)
    const Spec<float> sp = spec_of<float>(p, L, ws, true);
    const Cx<float>* tw = reinterpret_cast<const Cx<float>*>(ws + L.tw_y);
    if (vb.y == 0)
        ypass_body<float, true, ST_ANY>(reinterpret_cast<Cx<float>*>(ws + L.W), p.nx, p.ny, p.My, p.Mz / 2 + 1, p.ry, tw,
                                B.fft_tky, st, vb, sp.W3, sp.dy);
    else
        ypass_body<float, true, ST_ANY>(sp.W2, p.nx, p.ny, p.My, p.Mz / 2 + 1, p.ry, tw, B.fft_tky, st, vb);
}

__global__ void __launch_bounds__(FFT_THREADS<float>, FFT_MINB) kb_xconv(const BatchBeam* __restrict__ beams,
                                                        const int* __restrict__ start, int nb) {
    pdl_wait();
    BATCH_BEAM(BS_FFT_X)
    const Spec<float> sp = spec_of<float>(p, L, ws, true);
    xconv_body<float, ST_ANY>(reinterpret_cast<Cx<float>*>(ws + L.W), reinterpret_cast<const float*>(ws + L.green), p.nx,
                      p.My, p.Mz / 2 + 1, p.My / 2 + 1, p.rx, reinterpret_cast<const Cx<float>*>(ws + L.tw_x),
                      B.fft_tkx, st, vb, sp.W2, sp.dx);
}

// inverse z pass: block group f writes output f (the potential; with spectral
// fields also Ex, Ey, Ez), as k_zinv's blockIdx.z
__global__ void __launch_bounds__(FFT_THREADS<float>, FFT_MINB) kb_zinv(const BatchBeam* __restrict__ beams,
                                                       const int* __restrict__ start, int nb) {
    pdl_wait();
    BATCH_BEAM(BS_FFT_ZI)
    const Spec<float> sp = spec_of<float>(p, L, ws, true, false);
    const int f = vb.y / p.nx + sp.f0;
    const VBlk v = {vb.x, vb.y - (f - sp.f0) * p.nx, vb.nx, p.nx};
    const Cx<float>* src;
    float* out;
    const Cx<float>* dz;
    float mul;
    inv_out<float>(sp, st, f, reinterpret_cast<const Cx<float>*>(ws + L.W), reinterpret_cast<float*>(ws + L.phi), src,
                   out, dz, mul);
    zinv_body<float>(src, out, p.ny, p.nz, p.My, p.Mz / 2 + 1, p.rz, reinterpret_cast<const Cx<float>*>(ws + L.tw_z),
                     B.fft_nc, st, v, dz, mul, f - 1, p.nx);
}

__global__ void kb_field_octs(const BatchBeam* __restrict__ beams, const int* __restrict__ start, int nb) {
    pdl_wait();
    BATCH_BEAM(BS_FIELD)
    if (p.spectral)
        field_octs_spectral_body(reinterpret_cast<const float*>(ws + L.ex), reinterpret_cast<const float*>(ws + L.ey),
                                 reinterpret_cast<const float*>(ws + L.ez), reinterpret_cast<float*>(ws + L.exq),
                                 reinterpret_cast<float*>(ws + L.eyq), reinterpret_cast<float*>(ws + L.ezq), p.nx, p.ny,
                                 p.nz, st, vb);
    else
        field_octs_body(reinterpret_cast<const float*>(ws + L.phi), reinterpret_cast<float*>(ws + L.exq),
                        reinterpret_cast<float*>(ws + L.eyq), reinterpret_cast<float*>(ws + L.ezq), p.nx, p.ny, p.nz,
                        st, vb);
}
#undef BATCH_BEAM

// A batched launch gives every block the largest dynamic shared memory of
// its beams, so one beam with long lines would set the occupancy of all the
// others: the batch caps each beam's strided-pass blocks at what lets four
// blocks share an SM (228 KB per SM, 1 KB reserved per block).
constexpr size_t BATCH_FFT_SMEM = 233472 / 4 - 1024;
template <typename F>
static int batch_cols(int tk, F&& smem) {
    while (tk > 2 && smem(tk) > BATCH_FFT_SMEM) tk /= 2;
    return tk;
}

void batch_fft_tiling(BatchBeam& B, size_t smem[3]) {
    const Plan& p = B.p;
    const int Kz = p.Mz / 2 + 1;
    const int nbuf = p.spectral ? 3 : 2;  // line buffers of the x pass and the y passes
    B.fft_nc = z_lines_per_block(p.Mz);
    auto smem_y = [&](int tk) {
        const size_t f = smem_yf<float>(p.My, tk), i = smem_yi<float>(p.My, tk, p.spectral);
        return f > i ? f : i;
    };
    auto smem_xx = [&](int tk) { return smem_x<float>(p.Mx, tk, p.spectral); };
    B.fft_tky = batch_cols(pass_cols<float>(p.fft_cols_y, p.My, nbuf), smem_y);
    B.fft_tkx = batch_cols(pass_cols<float>(p.fft_cols_x, p.Mx, nbuf), smem_xx);
    B.gx[BS_FFT_Z] = (p.ny + 2 * B.fft_nc - 1) / (2 * B.fft_nc);
    B.gy[BS_FFT_Z] = p.nx;
    B.gx[BS_FFT_Y] = (p.nx * Kz + B.fft_tky - 1) / B.fft_tky;  // columns (x, kz)
    B.gy[BS_FFT_Y] = 1;
    B.gx[BS_FFT_X] = (p.My * Kz + B.fft_tkx - 1) / B.fft_tkx;  // columns (ky, kz)
    B.gy[BS_FFT_X] = 1;
    B.gx[BS_FFT_YI] = B.gx[BS_FFT_Y];
    B.gy[BS_FFT_YI] = p.spectral ? 2 : 1;
    B.gx[BS_FFT_ZI] = B.gx[BS_FFT_Z];
    B.gy[BS_FFT_ZI] = p.nx * (p.spectral ? 3 : 1);  // spectral fields: Ex, Ey, Ez (no potential)
    B.gx[BS_FIELD] = p.ny;
    B.gy[BS_FIELD] = p.nx;
    smem[0] = smem_zi<float>(p.Mz, B.fft_nc);
    if (smem_zf<float>(p.Mz, B.fft_nc) > smem[0]) smem[0] = smem_zf<float>(p.Mz, B.fft_nc);
    smem[1] = smem_y(B.fft_tky);
    smem[2] = smem_xx(B.fft_tkx);
}

cudaError_t prepare_batch_fft() {
    cudaError_t e;
    const size_t big = 48 * 1024 + 1;
    if ((e = smem_opt_in(reinterpret_cast<const void*>(kb_zfwd), big))) return e;
    if ((e = smem_opt_in(reinterpret_cast<const void*>(kb_yfwd), big))) return e;
    if ((e = smem_opt_in(reinterpret_cast<const void*>(kb_yinv), big))) return e;
    if ((e = smem_opt_in(reinterpret_cast<const void*>(kb_xconv), big))) return e;
    return smem_opt_in(reinterpret_cast<const void*>(kb_zinv), big);
}

// blocks: the five passes' block counts (z, y, x forward; y, z inverse)
cudaError_t launch_batch_convolve(const BatchBeam* beams, const int* sz, const int* sy, const int* sx,
                                  const int* syi, const int* szi, int nb, const int blocks[5], const size_t smem[3],
                                  cudaStream_t s, int part) {
    if (nb <= 0) return cudaSuccess;
    if (part != CONV_REST) {
        launch(kb_zfwd, blocks[0], FFT_THREADS<float>, smem[0], s, beams, sz, nb);
        launch(kb_yfwd, blocks[1], FFT_THREADS<float>, smem[1], s, beams, sy, nb);
    }
    if (part == CONV_FORWARD) return cudaGetLastError();
    launch(kb_xconv, blocks[2], FFT_THREADS<float>, smem[2], s, beams, sx, nb);
    launch(kb_yinv, blocks[3], FFT_THREADS<float>, smem[1], s, beams, syi, nb);
    launch(kb_zinv, blocks[4], FFT_THREADS<float>, smem[0], s, beams, szi, nb);
    return cudaGetLastError();
}

cudaError_t launch_batch_field(const BatchBeam* beams, const int* start, int nb, int blocks, cudaStream_t s) {
    if (nb <= 0) return cudaSuccess;
    launch(kb_field_octs, blocks, 128, 0, s, beams, start, nb);
    return cudaGetLastError();
}

}  // namespace ocsc
