// Lines of the FP64 transforms on the host: the steps of sc_dft.cuh in block
// fixed point and the same DFTs in double, each against extended precision.
// Prints "name L double-error fixed-error", errors in the 2-norm over the
// reference's, averaged over lines; "conversions <mismatches>".
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#define __device__
#define __host__
#define __forceinline__ inline
#define __align__(n) alignas(n)
struct float2 { float x, y; };
struct double2 { double x, y; };
static unsigned long long bits(double d) { unsigned long long b; memcpy(&b, &d, 8); return b; }
static int __double2hiint(double d) { return (int)(bits(d) >> 32); }
static int __double2loint(double d) { return (int)bits(d); }
static double __hiloint2double(int h, int l) {
    const unsigned long long b = ((unsigned long long)(unsigned)h << 32) | (unsigned)l;
    double d;
    memcpy(&d, &b, 8);
    return d;
}
static int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
static int __clzll(long long v) { return v ? __builtin_clzll((unsigned long long)v) : 64; }
using std::max;
#include "sc_dft.cuh"
using namespace ocsc;

typedef long double LD;
struct Z { LD x, y; };
typedef std::vector<double2> Line;

static Z root(int L, long m) {
    const LD a = 2 * acosl(-1.0L) * (m % L) / L;
    return {cosl(a), sinl(a)};
}
static std::vector<Z> dft(const std::vector<Z>& in, int sign) {
    const int L = (int)in.size();
    std::vector<Z> w(L), out(L, Z{0, 0});
    for (int i = 0; i < L; ++i) w[i] = root(L, i);
    for (int k = 0; k < L; ++k)
        for (int n = 0; n < L; ++n) {
            const Z c = w[(long)n * k % L];
            const LD s = sign * c.y;
            out[k].x += in[n].x * c.x - in[n].y * s;
            out[k].y += in[n].x * s + in[n].y * c.x;
        }
    return out;
}
static FxW fxw(int L, long m) { const Z c = root(L, m); return {FxC((double)c.x), FxC((double)-c.y)}; }
static double2 dw(int L, long m) { const Z c = root(L, m); return {(double)c.x, (double)-c.y}; }

// the forward steps in double (the line is zero from L / 2 on)
template <int L>
static Line fwd_double(const Line& in) {
    constexpr int Q = two_step_q(L), P = L / Q;
    Line t(L), out(L);
    for (int m = 0; m < Q; ++m) {
        double2 v[P];
        for (int n = 0; n < P; ++n) v[n] = in[n * Q + m];
        dft_reg<double, false, P, HALF_IN>(v);
        for (int k = 0; k < P; ++k) t[k * Q + m] = k ? twmul<double, false>(v[k], dw(L, (long)k * m)) : v[k];
    }
    for (int k = 0; k < P; ++k) {
        double2 u[Q];
        for (int n = 0; n < Q; ++n) u[n] = t[k * Q + n];
        dft_reg<double, false, Q, DFT_FULL>(u);
        for (int n = 0; n < Q; ++n) out[k + P * n] = u[n];
    }
    return out;
}
// the inverse steps (the transposed flow, the first half of the results)
template <int L>
static Line inv_double(const Line& in) {
    constexpr int Q = two_step_q(L), P = L / Q;
    Line t(L), out(L / 2);
    for (int m = 0; m < P; ++m) {
        double2 v[Q];
        for (int n = 0; n < Q; ++n) v[n] = in[n * P + m];
        dft_reg<double, true, Q, DFT_FULL>(v);
        for (int k = 0; k < Q; ++k) t[m * Q + k] = k ? twmul<double, true>(v[k], dw(L, (long)k * m)) : v[k];
    }
    for (int k = 0; k < Q; ++k) {
        double2 u[P];
        for (int n = 0; n < P; ++n) u[n] = t[n * Q + k];
        dft_reg<double, true, P, HALF_OUT>(u);
        for (int n = 0; n < P / 2; ++n) out[k + Q * n] = u[n];
    }
    return out;
}

// the steps of the x pass (xconv_fx): forward, times G, inverse; G empty: only the inverse
template <int L>
struct Fixed {
    using S = FxSteps<L>;
    static constexpr int Q = S::Q, P = S::P, ROW = S::ROW;
    std::vector<Fx2> tab, X;
    std::vector<FxW> tw;
    Fixed() : tab(P * ROW), X(L), tw(L, FxW{FxC(0, 0), FxC(0, 0)}) {
        for (int i = 0; i < P; ++i)
            for (int j = 0; j < Q; ++j) tw[i * Q + j] = fxw(L, (long)i * j);
    }
    static int exponent(const Line& in) {
        int E = 1;
        for (const double2& c : in) E = max(E, max(fx_exp(c.x), fx_exp(c.y)));
        return E;
    }
    template <int BIT>
    static Fx2 from(double2 c, int E) { return cx<Fx>(fx_from<BIT>(c.x, E), fx_from<BIT>(c.y, E)); }
    // forward into X; returns the bit of 2^E
    int forward(const Line& in, int E) {
        unsigned mag = 0;
        for (int m = 0; m < Q; ++m) {
            Fx2 v[P];
            for (int n = 0; n < P; ++n) v[n] = from<S::B_HALF>(in[n * Q + m], E);
            mag = max(mag, S::template first<false, HALF_IN>(v, m, tw.data(), tab.data()));
        }
        const int sh = fx_room<Q>(mag);
        for (int k1 = 0; k1 < P; ++k1) {
            Fx2 u[Q];
            S::template second<false>(u, k1, tab.data(), sh);
            for (int k2 = 0; k2 < Q; ++k2) X[k1 + P * k2] = u[k2];
        }
        return S::B_HALF - sh;
    }
    Line inverse(int E, int bit) {
        unsigned mag = 0;
        for (int n1 = 0; n1 < P; ++n1) {
            Fx2 v[Q];
            for (int n2 = 0; n2 < Q; ++n2) v[n2] = X[n1 + P * n2];
            mag = max(mag, S::t_first(v, n1, tw.data(), tab.data()));
        }
        const int sh = fx_room<P>(mag);
        const FxOut o(E, bit - sh);
        Line out(L / 2);
        for (int k2 = 0; k2 < Q; ++k2) {
            Fx2 u[P];
            S::t_second(u, k2, tab.data(), sh);
            for (int k1 = 0; k1 < P / 2; ++k1) out[k1 * Q + k2] = {fx_to(u[k1].x, o), fx_to(u[k1].y, o)};
        }
        return out;
    }
    Line pass(const Line& in, const std::vector<double>& G) {
        const int E = exponent(in);
        int bit = forward(in, E), top = 0;
        std::vector<int> e(L);
        for (int k = 0; k < L; ++k) {
            const FxC c = fx_fraction(G[k], e[k]);
            X[k] = cx<Fx>(fx_mul(X[k].x, c), fx_mul(X[k].y, c));
            top = max(top, fx_top(X[k], e[k]));
        }
        const int EG = top - (fx_bit(Q) + 1);
        for (int k = 0; k < L; ++k) X[k] = fx_scale(X[k], EG - e[k]);
        return inverse(E, bit - (EG - 1022));
    }
    Line fwd(const Line& in) {
        const int E = exponent(in), bit = forward(in, E);
        const FxOut o(E, bit);
        Line out(L);
        for (int k = 0; k < L; ++k) out[k] = {fx_to(X[k].x, o), fx_to(X[k].y, o)};
        return out;
    }
    Line inv(const Line& in) {
        const int E = exponent(in);
        for (int k = 0; k < L; ++k) X[k] = from<S::B_INV>(in[k], E);
        return inverse(E, S::B_INV);
    }
};

static std::vector<Z> wide(const Line& in) {
    std::vector<Z> out(in.size());
    for (size_t i = 0; i < in.size(); ++i) out[i] = {in[i].x, in[i].y};
    return out;
}
static LD error(const Line& a, const std::vector<Z>& ref) {
    LD d = 0, n = 0;
    for (size_t i = 0; i < a.size(); ++i) {
        d += (a[i].x - ref[i].x) * (a[i].x - ref[i].x) + (a[i].y - ref[i].y) * (a[i].y - ref[i].y);
        n += ref[i].x * ref[i].x + ref[i].y * ref[i].y;
    }
    return sqrtl(d / n);
}

template <int L>
static void lines() {
    std::mt19937_64 g(L);
    std::normal_distribution<double> N;
    std::uniform_real_distribution<double> U(0, 1);
    const int reps = 24;
    const char* what[] = {"random", "bunch", "alternating", "uniform alternating", "spike", "decades"};
    for (int kind = 0; kind < 6; ++kind) {
        LD fd = 0, ff = 0, id = 0, fi = 0, xd[3] = {0, 0, 0}, xf[3] = {0, 0, 0};
        const double kappa[3] = {1e-2, 1e-1, 1.0};  // G = 1 / (k^2 + kappa^2), as the Green's spectrum along a line
        for (int rep = 0; rep < reps; ++rep) {
            Line in(L, double2{0, 0});
            for (int i = 0; i < L / 2; ++i) {
                const double z = (i - L / 4) / (L / 10.), sc = exp(-z * z / 2), s = i & 1 ? -1 : 1;
                if (kind == 0) in[i] = {N(g), N(g)};
                if (kind == 1) in[i] = {sc * (1 + .1 * N(g)), sc * (1 + .1 * N(g))};
                if (kind == 2) in[i] = {s * sc, s * sc * .3};
                if (kind == 3) in[i] = {s * (1 + 1e-3 * N(g)), .5 * s};
                if (kind == 4 && i == rep % (L / 2)) in[i] = {1.37, -.7};
                if (kind == 5) in[i] = {N(g) * pow(10, -20 * U(g)), N(g) * pow(10, -20 * U(g))};
            }
            Fixed<L> F;
            const std::vector<Z> X = dft(wide(in), -1);
            fd += error(fwd_double<L>(in), X);
            ff += error(F.fwd(in), X);
            Line full(L);  // an inverse line: any spectrum
            for (int k = 0; k < L; ++k) full[k] = {(double)X[k].x, (double)X[k].y};
            if (kind == 4) { full.assign(L, double2{0, 0}); full[rep] = {1.37, -.7}; }
            const std::vector<Z> x = dft(wide(full), 1);
            id += error(inv_double<L>(full), x);
            fi += error(F.inv(full), x);
            for (int j = 0; j < 3; ++j) {
                std::vector<double> G(L);
                std::vector<Z> XG(L);
                Line D = fwd_double<L>(in);
                for (int k = 0; k < L; ++k) {
                    const double s = 2 * sin(acos(-1.0) * k / L);
                    G[k] = 1 / (s * s + kappa[j] * kappa[j]);
                    XG[k] = {X[k].x * G[k], X[k].y * G[k]};
                    D[k] = {D[k].x * G[k], D[k].y * G[k]};
                }
                const std::vector<Z> r = dft(XG, 1);
                xd[j] += error(inv_double<L>(D), r);
                xf[j] += error(F.pass(in, G), r);
            }
        }
        printf("forward,%s,%d,%.3Le,%.3Le\n", what[kind], L, fd / reps, ff / reps);
        printf("inverse,%s,%d,%.3Le,%.3Le\n", what[kind], L, id / reps, fi / reps);
        for (int j = 0; j < 3; ++j)
            printf("x pass %g,%s,%d,%.3Le,%.3Le\n", kappa[j], what[kind], L, xd[j] / reps, xf[j] / reps);
    }
}

// whether d is a nearest double of v
static bool nearest(double d, LD v) {
    return fabsl(v - d) <= fabsl(v - nextafter(d, -INFINITY)) && fabsl(v - d) <= fabsl(v - nextafter(d, INFINITY));
}

int main() {
    lines<64>();
    lines<96>();
    lines<128>();
    lines<192>();
    lines<256>();
    // conversions: any value, any line exponent above its own, denormals among both
    std::mt19937_64 g(5);
    long bad = 0;
    for (int i = 0; i < 1000000; ++i) {
        const long long v = (long long)g() >> (2 + g() % 62);
        const int E = 1 + (int)(g() % 2000);
        bad += !nearest(fx_to(Fx{v}, FxOut(E, 54)), ldexpl((LD)v, E - 1023 - 54));
        bad += !nearest(fx_double(Fx{v}), (LD)v);
        const double x = ldexp((double)(long long)g(), (int)(g() % 80) - (g() & 1 ? 100 : 1160));
        const int EE = max(fx_exp(x), 1) + (int)(g() % 70);
        const LD r = floorl(fabsl(ldexpl((LD)x, 1023 - EE + 54)) + 0.5L);
        bad += fx_from<54>(x, EE).v != (long long)(x < 0 ? -r : r);
    }
    printf("conversions,%ld\n", bad);
}
