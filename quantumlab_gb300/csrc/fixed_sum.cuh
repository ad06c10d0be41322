// fixed_sum.cuh -- sums of products of doubles on the integer pipes.
//
// A reduction of squares or products is bound by GB300's FP64 pipe (two
// operations an amplitude for a norm: 70 us at 24 qubits, HBM 39).  Values are
// aligned to the largest exponent E of a group as integers below 2^54, split
// into 27-bit digits, and their products summed in 64 bits; only a group's
// total becomes a double.  An aligned value is within 2^-55 of the group's
// largest, so a product's error is below the rounding of an FP64
// multiply-add on the group's largest product.  Groups are the four amplitudes
// of a thread's item.  On a dense state of 26 qubits, the whole call (HBM floors
// 158, 79, 316): total probability 319 us -> 203, probability of one outcome 174
// -> 116, inner product 615 -> 500.
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
// the same with x's sign
__device__ __forceinline__ int2 digits(double x, int E) {
    const int s = (__double2hiint(x) >> 31) | 1;
    const int2 d = absDigits(x, E);
    return make_int2(d.x * s, d.y * s);
}
__device__ __forceinline__ int64_t mad(int a, int b, int64_t c) { return c + (int64_t)a * b; }

struct Sums {                                    // h h, h l + l h, l l; at most 2^8 products
    int64_t hh, x, ll;
    __device__ __forceinline__ void add(int2 a, int2 b) {
        hh = mad(a.x, b.x, hh);
        x = mad(a.x, b.y, x);
        x = mad(a.y, b.x, x);
        ll = mad(a.y, b.y, ll);
    }
    // acc + c times the sum, in units of 2^54
    __device__ __forceinline__ double into(double acc, double c) const {
        return fma(c, (double)hh, fma(c * 0x1p-27, (double)(x + ((ll + (1 << 26)) >> 27)), acc));
    }
    // the sum of at most 16 products, rounded to units of 2^49
    __device__ __forceinline__ double few() const { return (double)((hh << 5) + ((x + (ll >> 27) + (1 << 21)) >> 22)); }
};
// 2^(a + b - 2103): the unit of few() for values aligned to exponents a and b;
// valid (a normal number) for the exponents that unitFits takes
__device__ __forceinline__ double unit(int a, int b) { return __hiloint2double((a + b - 1080) << 20, 0); }
__device__ __forceinline__ bool unitFits(int a, int b) { return a + b > 1080 && a + b < 3000 && max(a, b) < 0x7FF; }

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
