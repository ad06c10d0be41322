// ScaleInt against the FP64 product, bit for bit; prints the number of
// mismatches and of products that took the integer path's range.
#include "scale_int.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

static uint64_t bits(double x) {
    uint64_t u;
    memcpy(&u, &x, 8);
    return u;
}

int main() {
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> unit(0.0, 1.0);
    long wrong = 0, inRange = 0;
    const double fixed[] = {1.0, 0.5, 0.75, std::nextafter(1.0, 0.0), std::nextafter(0.5, 1.0), std::sqrt(0.98), 1.0 / 3, 1e-3, 0.0, -0.5, 1.5, 1e-200};
    const double odd[] = {0.0, -0.0, 1.0, -1.0, INFINITY, -INFINITY, 4.9e-324, 2.2250738585072014e-308, 1e308, 1e-200, 3.0, 1 + 0x1p-52};
    for (int k = 0; k < 400; ++k) {
        const double c = k < 12 ? fixed[k] : k < 200 ? unit(g) : std::ldexp((double)(g() >> 40), -24);   // short factors: ties
        const qg::ScaleInt s(c);
        for (int i = 0; i < 20000; ++i) {
            double x = i < 12 ? odd[i] : std::ldexp(unit(g) - 0.5, (int)(g() % 120) - 100);
            if (i % 7 == 0) x = std::ldexp((double)(int64_t)(g() >> (11 + g() % 30)), -60);           // few bits: ties and exact products
            inRange += x != 0;
            if (bits(s(x)) != bits(x * c)) ++wrong;
        }
    }
    const qg::ScaleInt s(0.5);
    if (!std::isnan(s(NAN))) ++wrong;
    printf("wrong %ld\nproducts %ld\n", wrong, inRange);
    return 0;
}
