// scale_int.cuh -- a double times a constant of (0, 1], rounded as the FP64
// product is, on the integer pipes (GB300's FP64 pipe executes two
// instructions a clock and SM).
//
// The functions compile for the device and, for the CPU unit test, for the
// host.
#pragma once

#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define QG_SI_HD __host__ __device__ __forceinline__
#else
#define QG_SI_HD inline
#endif

namespace qg {

#if defined(__CUDACC__)
static __host__ __device__ __noinline__ double scaleFp64(double x, double c) { return x * c; }
#else
inline double scaleFp64(double x, double c) { return x * c; }
#endif

struct ScaleInt {
    uint64_t m;          // c's 53 significant bits, leading one at bit 63; 0: c is not in the form's range
    int e;               // c's exponent field
    double c;

    explicit ScaleInt(double factor) : m(0), e(0), c(factor) {
        uint64_t u;
        memcpy(&u, &factor, 8);
        e = (int)(u >> 52);
        if (factor <= 1.0 && factor >= 0x1p-500) m = ((u & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) << 11;
    }

    QG_SI_HD double operator()(double x) const {
        uint64_t u;
#if defined(__CUDA_ARCH__)
        u = (uint64_t)__double_as_longlong(x);
#else
        memcpy(&u, &x, 8);
#endif
        const int ex = (int)(u >> 52) & 0x7FF;
        // zeros, subnormals, infinities, NaNs, results near the smallest: FP64
        if ((unsigned)(ex - 600) >= 0x7FFu - 600u || m == 0) return scaleFp64(x, c);
        const uint64_t mx = (u << 11) | 0x8000000000000000ull;
        uint64_t hi, lo;
#if defined(__CUDA_ARCH__)
        hi = __umul64hi(mx, m);
        lo = mx * m;
#else
        const unsigned __int128 w = (unsigned __int128)mx * m;
        hi = (uint64_t)(w >> 64);
        lo = (uint64_t)w;
#endif
        // (hi : lo) / 2^126 in [1, 4): the leading one to bit 63
        const uint32_t two = (uint32_t)(hi >> 63);
        if (!two) {
            hi = (hi << 1) | (lo >> 63);
            lo <<= 1;
        }
        // nearest, ties to even: the 11 bits below, and whether anything follows
        const uint64_t mant = hi >> 11;
        const uint32_t t = (((uint32_t)hi & 0x7FFu) << 1) | (lo != 0 ? 1u : 0u);
        const uint32_t up = (t + ((uint32_t)mant & 1u) + 0x7FFu) >> 12;
        const uint64_t r = ((uint64_t)(uint32_t)(ex + e - 1023 + (int)two - 1) << 52) + mant + up;
        u = (u & 0x8000000000000000ull) | r;
#if defined(__CUDA_ARCH__)
        return __longlong_as_double((long long)u);
#else
        memcpy(&x, &u, 8);
        return x;
#endif
    }
};

}  // namespace qg
