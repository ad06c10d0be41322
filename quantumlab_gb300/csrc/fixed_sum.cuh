// fixed_sum.cuh -- sums of products of doubles on the integer pipes.
//
// A reduction of squares or products is bound by GB300's FP64 pipe (two
// operations an amplitude for a norm: 70 us at 24 qubits, HBM 39).  Values are
// aligned to the largest exponent E of a group as integers, split into two
// digits, and their products summed in 64 bits; only a group's total becomes a
// double.
//   * Squares: integers below 2^54 in groups of four amplitudes.  The largest
//     value's square is in the sum, so an error of 2^-55 of that value is below
//     the rounding of an FP64 multiply-add on the sum.
//   * Products of two states: the largest values of either may meet small ones
//     only (nearly orthogonal states), so that their products all lie far below
//     the range of the aligned integers.  Groups are two amplitudes, integers
//     below 2^60, and a group whose largest product lies more than 2^5 below
//     the product of the two states' largest values takes FP64 (productsFit).
// On a dense state of 26 qubits, the whole call (HBM floors 158, 79, 316): total
// probability 319 us -> 203, probability of one outcome 174 -> 116, inner
// product 615 -> 550.
#pragma once

#include <stdint.h>

namespace qg {
namespace fsum {

// exponent field of the largest of some values, from the high words
__device__ __forceinline__ uint32_t magnitude(double x) { return (uint32_t)__double2hiint(x) & 0x7FFFFFFFu; }

// |x| 2^(1076 - E) rounded to an integer below 2^54, as h 2^27 + l.  (Not
// through fabs, which is an instruction of the FP64 pipe: eight of them an item
// left the norm of a dense state at 26 qubits FP64-bound, 338 us; 213 without.)
__device__ __forceinline__ int2 absDigits(double x, int E) {
    const uint32_t hi = (uint32_t)__double2hiint(x);
    const int e = (int)(hi >> 20) & 0x7FF;
    const uint64_t m = ((uint64_t)((hi & 0xFFFFFu) | (e ? 0x100000u : 0u)) << 32) | (uint32_t)__double2loint(x);
    uint64_t t;                                  // the shift gives 0 from 64 up
    asm("shr.u64 %0, %1, %2;" : "=l"(t) : "l"(m << 11), "r"(E - max(e, 1) + 9));
    t = (t + 1) >> 1;
    return make_int2((int)(t >> 27), (int)((uint32_t)t & 0x7FFFFFFu));
}
// x 2^(1082 - E) rounded to an integer below 2^60 in magnitude, as h 2^30 + l
__device__ __forceinline__ int2 wideDigits(double x, int E) {
    const uint32_t hi = (uint32_t)__double2hiint(x);
    const int e = (int)(hi >> 20) & 0x7FF, s = ((int)hi >> 31) | 1;
    const uint64_t m = ((uint64_t)((hi & 0xFFFFFu) | (e ? 0x100000u : 0u)) << 32) | (uint32_t)__double2loint(x);
    uint64_t t;
    asm("shr.u64 %0, %1, %2;" : "=l"(t) : "l"(m << 11), "r"(E - max(e, 1) + 3));
    t = (t + 1) >> 1;
    return make_int2((int)(t >> 30) * s, (int)((uint32_t)t & 0x3FFFFFFFu) * s);
}
__device__ __forceinline__ int64_t mad(int a, int b, int64_t c) { return c + (int64_t)a * b; }

struct Sums {                                    // h h, h l + l h, l l
    int64_t hh, x, ll;
    __device__ __forceinline__ void add(int2 a, int2 b) {
        hh = mad(a.x, b.x, hh);
        x = mad(a.x, b.y, x);
        x = mad(a.y, b.x, x);
        ll = mad(a.y, b.y, ll);
    }
    // the sum of at most 16 products, rounded to units of 2^49
    __device__ __forceinline__ double few() const { return (double)((hh << 5) + ((x + (ll >> 27) + (1 << 21)) >> 22)); }
    // the sum of at most 4 products of wide digits, rounded to units of 2^60
    __device__ __forceinline__ double wide() const { return (double)(hh + ((x + (ll >> 30) + (1 << 29)) >> 30)); }
};
// 2^(a + b - 2103): the unit of few() for values aligned to exponents a and b;
// valid (a normal number) for the exponents that unitFits takes
__device__ __forceinline__ double unit(int a, int b) { return __hiloint2double((a + b - 1080) << 20, 0); }
__device__ __forceinline__ bool unitFits(int a, int b) { return a + b > 1081 && a + b < 3000 && max(a, b) < 0x7FF; }
// 2^(a + b - 2104): the unit of wide()
__device__ __forceinline__ double wideUnit(int a, int b) { return __hiloint2double((a + b - 1081) << 20, 0); }

// Whether four products (sums of their factors' exponents: s0 to s3) keep FP64's
// precision as wide digits aligned to exponents E and F.  A rounded factor is
// off by at most 2^-60 of 2^E or 2^F, so a product by 2^-58 of 2^(E + F): 2^-53 of
// a product 2^5 below that, which is what FP64 rounds a product by.  A product
// with a zero factor is exact.  On a dense state one warp in 500 has a group
// that does not fit (2^4: one in 50, 2^3: one in 6).
constexpr int kWideSlack = 5;
__device__ __forceinline__ int exponentOf(uint32_t magnitude) { return magnitude ? (int)(magnitude >> 20) : -4096; }
__device__ __forceinline__ bool productsFit(int E, int F, int s0, int s1, int s2, int s3) {
    const int top = max(max(s0, s1), max(s2, s3));
    return top >= E + F - kWideSlack || top < 0;
}

__device__ __forceinline__ uint32_t lowWords(double2 a, double2 b) {
    return (uint32_t)(__double2loint(a.x) | __double2loint(a.y) | __double2loint(b.x) | __double2loint(b.y));
}

// sum of squares of eight values
static __device__ __noinline__ double squaresFp64(double2 a, double2 b, double2 c, double2 d) {
    return a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y + c.x * c.x + c.y * c.y + d.x * d.x + d.y * d.y;
}
// One warp in kFp64Share stays in FP64, so that both kinds of pipe work (after
// the zeros are told, which cost neither): the norm of a dense state at 26
// qubits 203, 217, 231 us with one in 4, 8 and none; inner products are best
// with none.
constexpr unsigned kFp64Share = 4;
__device__ __forceinline__ bool fp64Warp() { return ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) % kFp64Share == 0; }
// acc plus it
__device__ __forceinline__ double addSquares(double acc, double2 a, double2 b, double2 c, double2 d) {
    const double v[8] = {a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y};
    uint32_t top = 0, any = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        top = max(top, magnitude(v[k]));
        any |= (uint32_t)__double2loint(v[k]);
    }
    if ((top | any) == 0) return acc;
    const int E = (int)(top >> 20);
    if (!unitFits(E, E) || fp64Warp()) return acc + squaresFp64(a, b, c, d);
    int64_t hh = 0, x = 0, ll = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int2 t = absDigits(v[k], E);
        hh = mad(t.x, t.x, hh);
        x = mad(t.x, t.y, x);
        ll = mad(t.y, t.y, ll);
    }
    return fma(unit(E, E), Sums{hh, 2 * x, ll}.few(), acc);
}

}  // namespace fsum
}  // namespace qg
