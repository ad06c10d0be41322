// CPU check of the fixed-point maps of quantumlab_gb300/csrc/fix64.cuh
// (compiled by tests/test_fix64.py with g++; no GPU).  For orthogonal maps of
// the kinds that gates make and inputs of several spreads, prints the largest
// error beyond its bound and the mean square errors of the fixed-point and
// the FP64 chains against quadruple precision, in units of the result's last
// place.
#include "fix64.cuh"

#include <cmath>
#include <cstdio>
#include <random>

using namespace qg::fx;
#if __LDBL_MANT_DIG__ >= 113
typedef long double Quad;
#else
typedef __float128 Quad;
#endif

static std::mt19937_64 rng(20261205);
static double uniform() { return std::uniform_real_distribution<double>(-1, 1)(rng); }
static double gauss() { return std::normal_distribution<double>()(rng); }

// the real form of a random SU(2) gate (NT = 4) or a rotation (NT = 2) with
// every coefficient in range
static bool randomMap(double (&m)[4][4]) {
    double g[4], s = 0;
    for (double& v : g) v = gauss(), s += v * v;
    for (double& v : g) v /= std::sqrt(s);
    const double a = g[0], b = g[1], c = g[2], d = g[3];
    const double r[4][4] = {{a, -b, -c, -d}, {b, a, d, -c}, {c, -d, a, b}, {d, c, -b, a}};
    for (int i = 0; i < 16; ++i) m[i / 4][i % 4] = r[i / 4][i % 4];
    return true;
}
static bool randomMap(double (&m)[2][2]) {
    const double t = 3.141592653589793 * uniform();
    m[0][0] = m[1][1] = std::cos(t);
    m[1][0] = std::sin(t);
    m[0][1] = -m[1][0];
    return true;
}

template <int NT>
static void check(const char* name) {
    double excess = -1e300;
    long accepted = 0, refusedInputs = 0;
    for (int spread = 0; spread < 5; ++spread) {
        double sqFixed = 0, sqFp = 0;
        long count = 0;
        for (int i = 0; i < 400000; ++i) {
            double m[NT][NT], x[NT], y[NT];
            Map<NT> f;
            randomMap(m);
            if (!mapFits<NT>(m, f)) continue;
            ++accepted;
            for (int k = 0; k < NT; ++k) {
                const int down = spread == 0 ? 0 : (int)(rng() % (spread == 1 ? 8 : spread == 2 ? 30 : spread == 3 ? 70 : 200));
                x[k] = std::ldexp(gauss(), -down - (int)(rng() % 2) * 300 * (i % 3 == 0));
                if (spread >= 3 && rng() % 4 == 0) x[k] = 0;
            }
            double* p[NT];
            for (int k = 0; k < NT; ++k) y[k] = x[k], p[k] = &y[k];
            double* const(&pc)[NT] = p;
            if (!apply<NT>(f, pc)) {
                ++refusedInputs;
                continue;
            }
            double mx = 0;
            for (double v : x) mx = std::fmax(mx, std::fabs(v));
            int e;
            std::frexp(mx, &e);                                    // mx in [2^(e-1), 2^e)
            const double unit = std::ldexp(1.0, e - 1 - 59);
            for (int o = 0; o < NT; ++o) {
                Quad want = 0;
                for (int k = 0; k < NT; ++k) want += (Quad)m[o][k] * x[k];
                double chain = m[o][0] * x[0];
                for (int k = 1; k < NT; ++k) chain = std::fma(m[o][k], x[k], chain);
                int ey;
                std::frexp((double)want, &ey);
                const double ulp = std::ldexp(1.0, ey - 53);
                const double err = (double)((Quad)y[o] - want), errFp = (double)((Quad)chain - want);
                // truncated inputs (row sums <= 2) and the last half unit
                excess = std::fmax(excess, (std::fabs(err) - 0.5 * ulp * (1 + 1e-9)) / unit - 2.5);
                if ((double)want != 0) {
                    sqFixed += err / ulp * (err / ulp);
                    sqFp += errFp / ulp * (errFp / ulp);
                    ++count;
                }
            }
        }
        // cancelled results weigh most in both sums
        printf("%s_rms_fixed_%d %.6e\n%s_rms_fp64_%d %.6e\n", name, spread, std::sqrt(sqFixed / count), name, spread,
               std::sqrt(sqFp / count));
    }
    printf("%s_excess_units %.6e\n%s_accepted %ld\n%s_refused_inputs %ld\n", name, excess, name, accepted, name, refusedInputs);
}

int main() {
    check<4>("four");
    check<2>("two");
    // maps that must take FP64: a small coefficient, a zero, a row beyond an orthogonal one
    int kept = 0;
    Map<2> f2;
    const double small[2][2] = {{1, -0x1p-7}, {0x1p-7, 1}}, id[2][2] = {{1, 0}, {0, 1}}, big[2][2] = {{1, 1}, {1, 1.5}};
    const double nan[2][2] = {{0.6, -0.8}, {0.8, NAN}};
    kept += mapFits<2>(small, f2) + mapFits<2>(id, f2) + mapFits<2>(big, f2) + mapFits<2>(nan, f2);
    printf("unfit_maps_taken %d\n", kept);
    // inputs that must take FP64
    const double h[2][2] = {{0.6, -0.8}, {0.8, 0.6}};
    mapFits<2>(h, f2);
    int taken = 0;
    const double odd[][2] = {{0, 0}, {INFINITY, 1}, {1, NAN}, {1e-310, 0}, {0, 1.7e308}, {-0.0, 0}};
    for (auto& v : odd) {
        double a = v[0], b = v[1];
        double* const p[2] = {&a, &b};
        taken += apply<2>(f2, p);
    }
    printf("odd_inputs_taken %d\n", taken);
    // a zero or a subnormal beside an ordinary input, and the ends of the range
    double worst = 0;
    const double pairs[][2] = {{1, 0}, {0, -1}, {1e-320, 1}, {0x1p-958, 0}, {0x1.fp917, 1}, {1, 0x1p-1000}};
    for (auto& v : pairs)
        for (int k = 0; k < 2; ++k) {
            double a = v[k], b = v[1 - k];
            const double want0 = h[0][0] * a + h[0][1] * b, want1 = h[1][0] * a + h[1][1] * b;
            double* const p[2] = {&a, &b};
            if (!apply<2>(f2, p)) worst = 1;
            worst = std::fmax(worst, std::fmax(std::fabs(a - want0) / std::fabs(want0), std::fabs(b - want1) / std::fabs(want1)));
        }
    printf("edge_rel %.6e\n", worst);
    return 0;
}
