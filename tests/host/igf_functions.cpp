// Errors of the functions of sc_igf_fn.cuh in units in the last place of the
// exact value (extended precision): prints "name,range,largest error".
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>

#define __restrict__
using std::fma;
using std::sqrt;
#include "sc_igf_fn.cuh"
using namespace ocsc;

typedef long double LD;
static const LogEntry LT[] = {SC_IGF_LOG_TABLE};
static const AtanEntry AT[] = {SC_IGF_ATAN_TABLE};

static std::mt19937_64 g(1);
static double U() { return std::uniform_real_distribution<double>(0, 1)(g); }
static double ulps(double v, LD exact) {
    if (exact == 0) return v == 0 ? 0 : 1e300;
    int e;
    frexp((double)exact, &e);
    return (double)(fabsl(v - exact) / ldexpl(1, e - 53));
}
static double neighbour(double x) {  // x or one of the few doubles beside it
    for (int s = (int)(g() % 7) - 3; s; s += s > 0 ? -1 : 1) x = nextafter(x, s > 0 ? INFINITY : 0);
    return x;
}
template <typename F, typename E, typename G>
static void run(const char* name, const char* range, F&& f, E&& exact, G&& gen, int n = 400000) {
    double worst = 0;
    for (int i = 0; i < n; ++i) {
        double a, b = 1;
        gen(a, b);
        const double e = ulps(f(a, b), exact(a, b));
        if (!(e <= worst)) worst = e;
    }
    printf("%s,%s,%.4f\n", name, range, worst);
}

int main() {
    auto lg = [](double x, double) { return igf::log_(x, LT); };
    auto lge = [](double x, double) { return logl((LD)x); };
    run("log", "2^-180 .. 2^180", lg, lge, [](double& x, double&) { x = exp2(360 * U() - 180); });
    run("log", "2^-41 .. 2^41", lg, lge, [](double& x, double&) { x = exp2(82 * U() - 41); });
    run("log", "0.1 .. 10", lg, lge, [](double& x, double&) { x = exp(4.6 * U() - 2.3); });
    run("log", "0.98 .. 1.02", lg, lge, [](double& x, double&) { x = 0.98 + 0.04 * U(); });
    for (int j = 2; j <= 53; j += 3) {
        char r[32];
        snprintf(r, sizeof r, "1 +- 2^-%d", j);
        run("log", r, lg, lge, [j](double& x, double&) { x = 1 + ldexp(2 * U() - 1, -j); }, 50000);
    }
    run("log", "table intervals", lg, lge,
        [](double& x, double&) { x = neighbour(ldexp(1 + (int)(128 * U()) / 128.0, (int)(9 * U()) - 4)); });
    run("log", "1 +- 2^-8 (the end of the series about 1)", lg, lge,
        [](double& x, double&) { x = neighbour(g() & 1 ? 1 + 0x1p-8 : 1 - 0x1p-8); }, 1000);
    run("log", "1", lg, lge, [](double& x, double&) { x = 1; }, 1);

    auto at = [](double n, double d) { return igf::atan_(n, d, AT); };
    auto ate = [](double n, double d) { return atanl((LD)n / d); };
    auto quotient = [](double w, double& n, double& d) {
        d = exp2(40 * U() - 20) * (g() & 1 ? 1 : -1);
        n = w * d * (g() & 1 ? 1 : -1);
    };
    run("atan", "2^-100 .. 2^100", at, ate, [&](double& n, double& d) { quotient(exp2(200 * U() - 100), n, d); });
    run("atan", "2^-30 .. 2^30", at, ate, [&](double& n, double& d) { quotient(exp2(60 * U() - 30), n, d); });
    run("atan", "0.1 .. 10", at, ate, [&](double& n, double& d) { quotient(exp(4.6 * U() - 2.3), n, d); });
    run("atan", "3.5/128 (the switch to the quotient itself)", at, ate,
        [&](double& n, double& d) { quotient(3.5 / 128 * (1 + 1e-6 * (U() - .5)), n, d); });
    run("atan", "table intervals", at, ate,
        [&](double& n, double& d) { quotient((4 + (int)(124 * U()) + .5) / 128 * (1 + 1e-7 * (U() - .5)), n, d); });
    run("atan", "1", at, ate, [&](double& n, double& d) { quotient(neighbour(1), n, d); });

    run("sqrt", "2^-300 .. 2^300", [](double x, double) { return igf::sqrt_(x); }, [](double x, double) { return sqrtl((LD)x); },
        [](double& x, double&) { x = exp2(600 * U() - 300); });
    run("div", "2^-300 .. 2^300", [](double n, double d) { return igf::div_(n, d); },
        [](double n, double d) { return (LD)n / d; },
        [](double& n, double& d) { n = exp2(300 * U() - 150) * (g() & 1 ? 1 : -1); d = exp2(300 * U() - 150); });
}
