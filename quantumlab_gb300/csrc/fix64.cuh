// fix64.cuh -- real linear maps of a few doubles in 61-bit fixed point, for
// the plain path's gates.
//
// GB300 executes 1.7-2.0 FP64 operations per clock per SM, against 64
// 32 x 32 + 64-bit integer multiply-adds (both measured).  A general 2 x 2
// gate needs 8 FP64 multiply-adds per amplitude and so ran at 30 % of HBM
// bandwidth.  Here its outputs y_o = sum_k c_ok x_k (k < NT reals of one
// amplitude pair) are computed on the integer pipes, no less precisely:
//   * the NT inputs are aligned to the largest one's exponent E as integers
//     T = mantissa 2^7 >> (E - e) below 2^60: an input within 2^-7 of the
//     largest keeps all its bits, a smaller one loses what lies below the
//     unit, 2^-59 to 2^-60 of the largest;
//   * the coefficients are the integers c 2^61 (exact for |c| >= 2^-8), split
//     as h 2^31 + l with a centred l; an aligned input is split as
//     h 2^31 + l, both with x's sign;
//   * the digit products are summed in 64 bits (4 wide multiply-adds a
//     term), and the total, kept to half a unit, is converted to a double
//     with one rounding.
// Error of an output: half an ulp of the result, plus under one unit for
// every input that lost bits.  FP64's chain rounds once per term, each time
// to half an ulp of a partial sum.  The chain's error is the larger one
// unless the largest input meets a small coefficient and nothing else
// contributes, so a map qualifies (mapFits) when every |c| is at least 2^-6
// (NT = 4) or 2^-5 (NT = 2): at that coefficient the unit is at most a
// quarter (half) of the result's last place.  |c| <= 1 and row sums <= 2, as
// the orthogonal maps of unitary gates have them, keep the sums in 64 bits.
// Inputs whose largest exponent leaves no room for the result's exponent
// (|x| < 2^-959 or >= 2^958, infinities, NaNs) are told by `apply`; they take
// FP64 arithmetic instead.
//
// The functions compile for the device and, for the CPU unit test, for the
// host.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define QG_FX_HD __host__ __device__ __forceinline__
#else
#define QG_FX_HD inline
#endif

namespace qg {
namespace fx {

struct Digits {
    int32_t h, l;
};

// a coefficient 2^-8 <= |c| <= 1 as (h 2^31 + l) 2^-61, |l| <= 2^30
inline Digits coefficient(double c) {
    const int64_t v = (int64_t)(c * 0x1p61);               // exact
    const int64_t low = ((v + (1ll << 30)) & ((1ll << 31) - 1)) - (1ll << 30);
    return Digits{(int32_t)((v - low) >> 31), (int32_t)low};
}

// The map of NT inputs to NT outputs as coefficient digits; valid when fits.
template <int NT>
struct Map {
    Digits c[NT][NT];
};
template <int NT>
inline bool mapFits(const double (&m)[NT][NT], Map<NT>& out) {
    const double least = NT == 4 ? 0x1p-6 : 0x1p-5;
    for (int o = 0; o < NT; ++o) {
        double sum = 0;
        for (int k = 0; k < NT; ++k) {
            const double a = fabs(m[o][k]);
            if (!(a >= least && a <= 1.0 + 1e-9)) return false;
            sum += a;
            out.c[o][k] = coefficient(m[o][k]);
        }
        if (sum > 2.0 + 1e-9) return false;
    }
    return true;
}

QG_FX_HD void words(double d, uint32_t& hi, uint32_t& lo) {
#if defined(__CUDA_ARCH__)
    hi = (uint32_t)__double2hiint(d);
    lo = (uint32_t)__double2loint(d);
#else
    uint64_t u;
    memcpy(&u, &d, 8);
    hi = (uint32_t)(u >> 32);
    lo = (uint32_t)u;
#endif
}
QG_FX_HD double fromBits(uint64_t u) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)u);
#else
    double d;
    memcpy(&d, &u, 8);
    return d;
#endif
}
QG_FX_HD uint64_t shiftRight(uint64_t m, uint32_t d) {     // 0 from d = 64 up
#if defined(__CUDA_ARCH__)
    uint64_t r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(m), "r"(d));
    return r;
#else
    return d < 64 ? m >> d : 0;
#endif
}
QG_FX_HD int64_t mulAdd(int32_t a, int32_t b, int64_t c) {
#if defined(__CUDA_ARCH__)
    int64_t r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
#else
    return c + (int64_t)a * b;
#endif
}

// The exponent field of the largest input (hi: the high words).
template <int NT>
QG_FX_HD uint32_t largestExponent(const uint32_t (&hi)[NT]) {
    uint32_t m = hi[0] & 0x7FFFFFFFu;
    for (int k = 1; k < NT; ++k) {
        const uint32_t a = hi[k] & 0x7FFFFFFFu;
        m = a > m ? a : m;
    }
    return m >> 20;
}
// exponents for which every output's exponent stays in range
QG_FX_HD bool exponentFits(uint32_t E) { return E - 64u <= 1980u - 64u; }

// Digits of x aligned to exponent E (a zero or subnormal x is shifted out);
// h is 4 times the high digit (below 2^31), as dot takes it.
QG_FX_HD Digits align(uint32_t hi, uint32_t lo, uint32_t E) {
    const uint32_t e = (hi & 0x7FFFFFFFu) >> 20;
    const uint32_t mh = (((hi << 8) | (lo >> 24)) & 0x0FFFFFFFu) | 0x10000000u;
    const uint64_t t = shiftRight(((uint64_t)mh << 32) | (lo << 8), E - e);
    const int32_t s = ((int32_t)hi >> 31) | 1;
    return Digits{(int32_t)(t >> 32) * (s * 4), (int32_t)((uint32_t)t >> 1) * s};
}

// sum_k c_k x_k in half units (below 2^62).  Each digit order's sum is
// shifted into the start of the next one's, so a term is multiply-adds only.
template <int NT>
QG_FX_HD int64_t dot(const Digits (&c)[NT], const Digits (&x)[NT]) {
    int64_t s = 0;
    for (int k = 0; k < NT; ++k) s = mulAdd(x[k].l, c[k].l, s);
    s >>= 31;
    for (int k = 0; k < NT; ++k) {
        s = mulAdd(x[k].h >> 2, c[k].l, s);
        s = mulAdd(x[k].l, c[k].h, s);
    }
    s >>= 29;
    for (int k = 0; k < NT; ++k) s = mulAdd(x[k].h, c[k].h, s);
    return s;
}

// y 2^(E - 1083) as a double, rounded to nearest.  The conversion instruction
// runs on the FP64 pipe, at its rate.
QG_FX_HD double finish(int64_t y, uint32_t E) {
    uint32_t hi, lo;
#if defined(__CUDA_ARCH__)
    words(__ll2double_rn(y), hi, lo);
#else
    words((double)y, hi, lo);
#endif
    hi = hi == 0 ? 0 : hi + ((E - 1083u) << 20);
    return fromBits(((uint64_t)hi << 32) | lo);
}

// x <- m x; false (x unchanged) when the exponents are out of range
template <int NT>
QG_FX_HD bool apply(const Map<NT>& m, double* const (&x)[NT]) {
    uint32_t hi[NT], lo[NT];
    for (int k = 0; k < NT; ++k) words(*x[k], hi[k], lo[k]);
    const uint32_t E = largestExponent(hi);
    if (!exponentFits(E)) return false;
    Digits d[NT];
    for (int k = 0; k < NT; ++k) d[k] = align(hi[k], lo[k], E);
    for (int o = 0; o < NT; ++o) *x[o] = finish(dot(m.c[o], d), E);
    return true;
}

}  // namespace fx
}  // namespace qg
