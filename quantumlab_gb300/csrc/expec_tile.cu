// expec_tile.cu -- the expectation value of a Pauli sum on a state vector,
// many terms per pass over the state (sm_103a).
//
// One reduction per X/Y mask (reduce.cu) reads the state once per mask and
// spends 3 to 5 FP64 operations on a pair: at 24 qubits 151 us a mask and 501
// us for the diagonal terms, bound by the FP64 pipe, against 39 us of HBM
// time.  Here a block takes tiles of 2^b amplitudes into shared memory and adds
// up every mask that lies in the tile's qubits:
//   * Re or Im of conj(psi_j) psi_k in two FP64 multiply-adds, over the pairs
//     on which the mask's terms do not cancel (a quarter of the amplitudes for
//     X..X and Y..Y of equal weight); two terms a step, steps of equal weights
//     into one sum.  Warps whose pairs hold a zero each (particle-number
//     sectors leave most of a register zero) spend no FP64.  Integer products
//     against the tile's largest amplitude would be faster on dense states,
//     but lose the products that are far below it: <X> of (1, e) is e.
//   * all diagonal terms through one Walsh-Hadamard transform of the tile's
//     |psi|^2 in 64-bit integers, scaled so that the tile's sum fills them:
//     a term is then one entry, whatever its weight.  A value is rounded to
//     2^-55 of the tile's largest amplitude, a probability to 2^-62 of the
//     tile's sum: less than the rounding of FP64 sums of |psi|^2.
// Energy of a 12-site Hubbard chain (24 qubits, 22 masks and 36 diagonal terms),
// the whole call: 3.91 ms -> 0.64 ms on a state without zeros, 0.50 ms after a
// short evolution from a classical state; 16 qubits 147 -> 47 us.
#include "chain_launch.cuh"
#include "fixed_sum.cuh"
#include "pauli_expec.h"

#include <algorithm>
#include <cmath>

namespace qg {
namespace {

using fsum::absDigits;

constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kMaxTileBits = 12, kMinTileBits = 8;
constexpr int kLow = 3;                          // qubits 0..2 are tile qubits: runs of 64 bytes
constexpr int kMaxOps = 48, kMaxDiag = 128;

// Sum over pairs (j, j ^ x), j with bit `pair` clear, of (-1)^popc(j & m)
// c[popc(j & d) & 1] times Re (or Im) of conj(psi_j) psi_k
struct PairOp {
    double c[2];
    uint64_t m, d;               // the masks' qubits outside the tile
    uint32_t xl, ml, dl;         // tile qubits of x, m, d
    int pair;                    // the bit of xl that is clear in j: the highest, for lanes in a row
    int fix;                     // one parity has no weight: the tile bit of d that is set for the other, or -1
    int imag;
    int flush;                   // the next step has other weights
};
struct ExpecPass {
    int b, numOps, numDiag;
    unsigned char pos[kMaxTileBits];             // the tile's qubits, ascending
    PairOp op[kMaxOps];
    uint64_t dm[kMaxDiag];                       // diagonal terms: qubits outside the tile,
    uint32_t dml[kMaxDiag];                      // tile qubits,
    double dc[kMaxDiag];                         // weight
};

__device__ __forceinline__ uint32_t insert0(uint32_t k, int b) { return ((k >> b) << (b + 1)) | (k & ((1u << b) - 1u)); }

// Where entry i of the transform lies: rounds over bits 0-2 and 3-5 would meet
// in a few banks.
__device__ __forceinline__ uint32_t place(uint32_t i) { return i ^ ((i >> 3) & 15u); }

struct PairLoop {                                // a step on this tile
    uint32_t xl, ml, dl, outM, outD, pairs;
    int pair, fix, one;          // one: the parity that acts, -1: both
    bool skip;                   // pairs with a zero add nothing
};
__device__ __forceinline__ double flip(double v, uint32_t sign) {      // sign: 0 or 1
    return __hiloint2double(__double2hiint(v) ^ (int)(sign << 31), __double2loint(v));
}
__device__ __forceinline__ bool nonzero(double x, double y) {
    return (((uint32_t)__double2hiint(x) | (uint32_t)__double2hiint(y)) << 1 | (uint32_t)(__double2loint(x) | __double2loint(y))) != 0;
}
// Pair t's j is t with zeros inserted: a thread's part (its index) and the
// round's part, the same for all threads, are worked out apart, parities too.
// (pairs is a multiple of 32, so that a warp's lanes take part together.)
template <bool IMAG, bool BOTH>
__device__ __forceinline__ void addPairs(const PairLoop& o, const double* sr, const double* si, double& s0, double& s1) {
    if (threadIdx.x >= o.pairs) return;
    const bool fixed = o.fix >= 0;
    const int b0 = fixed ? min(o.pair, o.fix) : o.pair, b1 = fixed ? max(o.pair, o.fix) : 31;
    const uint32_t jt = insert0(insert0(threadIdx.x, b0), b1);
    const uint32_t parT = __popc(jt & o.dl), sgnT = __popc(jt & o.ml);
    const uint32_t fixM = fixed && (o.ml >> o.fix & 1u);         // the fixed bit is one of ml's
#pragma unroll 2
    for (uint32_t u = 0; u < o.pairs; u += kThreads) {
        const uint32_t ju = insert0(insert0(u, b0), b1);
        const uint32_t parU = __popc(ju & o.dl) ^ o.outD, sgnU = __popc(ju & o.ml) ^ o.outM;
        uint32_t j = jt | ju, par = (parT ^ parU) & 1u, sg = sgnT ^ sgnU;
        if (!BOTH && fixed) {
            const uint32_t f = par ^ (uint32_t)o.one;
            j |= f << o.fix;
            sg ^= f & fixM;
        }
        const uint32_t k = j ^ o.xl;
        const double jr = sr[j], ji = si[j], kr = sr[k], ki = si[k];
        // (a zero with an infinity or NaN is no zero)
        if (o.skip && !__any_sync(0xffffffffu, nonzero(jr, ji) && nonzero(kr, ki))) continue;
        sg &= 1u;
        const double x = flip(jr, sg), y = flip(ji, IMAG ? sg ^ 1u : sg);      // Im: jr ki - ji kr
        double& s = BOTH && par ? s1 : s0;
        s = fma(y, IMAG ? kr : ki, fma(x, IMAG ? ki : kr, s));
    }
}

// A block's sum of diagonal terms as an unevaluated pair (TwoSum, TwoProduct).
// They are few and each may be as large as the result: rounded one by one, on
// registers of 8 to 14 qubits the sum was 1.3 times as far off as a reduction
// per mask, so 0.3 times.
struct Pair {
    double hi, lo;
    __device__ __forceinline__ void add(double x) {
        const double s = hi + x, z = s - hi;
        lo += (hi - (s - z)) + (x - z);
        hi = s;
    }
    __device__ __forceinline__ void add(const Pair& p) {
        add(p.hi);
        lo += p.lo;
    }
    __device__ __forceinline__ void addProduct(double c, int64_t q) {
        const double x = (double)q, p = c * x;
        lo += fma(c, x, -p) + c * (double)(q - (int64_t)x);
        add(p);
    }
};
__device__ __forceinline__ double warpSum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

__global__ void __launch_bounds__(kThreads) kExpecTile(const double* re, const double* im,
                                                       uint64_t tiles, const __grid_constant__ ExpecPass p,
                                                       double* partials, unsigned* counter, double* result) {
    extern __shared__ double sm[];
    __shared__ int shE[kWarps];
    __shared__ float shS[kWarps];
    __shared__ double shD[kWarps];
    __shared__ Pair shP[kMaxDiag / 32];
    __shared__ bool amLast;
    const int b = p.b, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t size = 1u << b;
    double* sr = sm;
    double* si = sr + size;
    uint64_t* high = reinterpret_cast<uint64_t*>(si + size);             // qubits of tile index bits >= kLow
    for (uint32_t h = tid; h < size >> kLow; h += kThreads) {
        uint64_t a = 0;
        for (int k = kLow; k < b; ++k) a |= (uint64_t)((h >> (k - kLow)) & 1u) << p.pos[k];
        high[h] = a;
    }
    chainStart();
    Pair diag{0.0, 0.0};
    double acc = 0.0;                            // the pairs' sum
    for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        uint64_t base = tile;
        for (int k = 0; k < b; ++k) base = ((base >> p.pos[k]) << (p.pos[k] + 1)) | (base & ((1ull << p.pos[k]) - 1ull));
        __syncthreads();
        // the tile as it is, and its largest exponent
        int E = 1;
        for (uint32_t l = 2 * tid; l < size; l += 2 * kThreads) {
            const uint64_t a = base | high[l >> kLow] | (l & ((1u << kLow) - 1u));
            const double2 r = *reinterpret_cast<const double2*>(re + a), i = *reinterpret_cast<const double2*>(im + a);
            *reinterpret_cast<double2*>(sr + l) = r;
            *reinterpret_cast<double2*>(si + l) = i;
            const uint32_t w = max(max(__double2hiint(r.x) & 0x7FFFFFFF, __double2hiint(r.y) & 0x7FFFFFFF),
                                   max(__double2hiint(i.x) & 0x7FFFFFFF, __double2hiint(i.y) & 0x7FFFFFFF));
            E = max(E, (int)(w >> 20));
        }
        E = __reduce_max_sync(0xffffffffu, E);
        if (lane == 0) shE[warp] = E;
        __syncthreads();
        for (int w = 0; w < kWarps; ++w) E = max(E, shE[w]);
        double s0 = 0.0, s1 = 0.0;
        for (int o = 0; o < p.numOps; ++o) {
            const PairOp& op = p.op[o];
            PairLoop pl{op.xl, op.ml, op.dl, (uint32_t)__popcll(base & op.m) & 1u, (uint32_t)__popcll(base & op.d) & 1u, 0,
                        op.pair, op.fix, op.c[0] != 0 && op.c[1] != 0 ? -1 : op.c[0] != 0 ? 0 : 1, E != 0x7FF};
            const int one = pl.one;
            pl.pairs = pl.dl == 0 && one >= 0 && (int)pl.outD != one ? 0 : pl.fix >= 0 ? size / 4 : size / 2;
            if (op.imag) {
                if (one < 0) addPairs<true, true>(pl, sr, si, s0, s1);
                else addPairs<true, false>(pl, sr, si, s0, s1);
            } else {
                if (one < 0) addPairs<false, true>(pl, sr, si, s0, s1);
                else addPairs<false, false>(pl, sr, si, s0, s1);
            }
            if (op.flush) {
                acc = fma(op.c[0] != 0 ? op.c[0] : op.c[1], s0, acc);
                if (one < 0) acc = fma(op.c[1], s1, acc);
                s0 = s1 = 0.0;
            }
        }
        if (p.numDiag == 0) continue;
        if (E == 0x7FF) {                        // infinities or NaNs: so is the sum
            acc = __longlong_as_double(0x7FF8000000000000ll);
            continue;
        }
        __syncthreads();
        // |psi|^2 in units of 2^46 products, then scaled to the tile's sum
        int64_t* q = reinterpret_cast<int64_t*>(sr);
        float sum = 0.f;
        for (uint32_t l = tid; l < size; l += kThreads) {
            const int2 r = absDigits(sr[l], E), i = absDigits(si[l], E);
            const uint64_t x = ((uint64_t)r.x << 36) | ((uint64_t)r.y << 9), y = ((uint64_t)i.x << 36) | ((uint64_t)i.y << 9);
            const int64_t v = (int64_t)(__umul64hi(x, x) + __umul64hi(y, y) + ((x * x) >> 63) + ((y * y) >> 63));
            sum += __ll2float_ru(v);
            __syncwarp();                        // place(l) is in this warp's sixteen
            q[place(l)] = v;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) shS[warp] = sum;
        __syncthreads();
        sum = 0.f;
        for (int w = 0; w < kWarps; ++w) sum += shS[w];
        // sum < 2^(62 + shift), with room for the roundings
        int shift = max(0, (int)((__float_as_uint(sum * 1.01f) >> 23) & 0xFF) - 127 + 1 - 62);
        const int64_t half = shift ? 1ll << (shift - 1) : 0;
        for (int level = 0; level < b; level += 3) {                 // three bits at a time in registers
            const int bits = min(3, b - level);
            for (uint32_t g = tid; g < size >> 3; g += kThreads) {
                // eight entries: the bits of this round, and for a last round of
                // fewer the lowest bits too, left alone
                const uint32_t rest = level + 3 <= b ? ((g >> level) << (level + 3)) | (g & ((1u << level) - 1u)) : 0;
                uint32_t at[8];
                int64_t v[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    at[k] = level + 3 <= b ? rest | ((uint32_t)k << level)
                                           : ((uint32_t)(k & ((1 << bits) - 1)) << level) | (g << (3 - bits)) | (uint32_t)(k >> bits);
                    at[k] = place(at[k]);
                    v[k] = q[at[k]];
                    if (level == 0) v[k] = (v[k] + half) >> shift;
                }
#pragma unroll
                for (int sb = 1; sb < 8; sb <<= 1) {
                    if (sb >> bits) break;
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (!(k & sb)) {
                            const int64_t x = v[k], y = v[k | sb];
                            v[k] = x + y;
                            v[k | sb] = x - y;
                        }
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) q[at[k]] = v[k];
            }
            __syncthreads();
        }
        const double pu = scalbn(1.0, 2 * E - 2106 + shift);
        for (int t = tid; t < p.numDiag; t += kThreads) {
            const double c = (__popcll(base & p.dm[t]) & 1) ? -p.dc[t] : p.dc[t];
            diag.addProduct(c * pu, q[place(p.dml[t])]);
        }
    }
    // block and grid sums in a fixed order, as in reduce_kernel.cuh
    acc = warpSum(acc);
    if (lane == 0) shD[warp] = acc;
    if (32 * warp < p.numDiag) {                 // (the threads that hold terms)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            diag.add(Pair{__shfl_down_sync(0xffffffffu, diag.hi, o), __shfl_down_sync(0xffffffffu, diag.lo, o)});
        if (lane == 0) shP[warp] = diag;
    }
    __syncthreads();
    if (tid == 0) {
        Pair v{0.0, 0.0};
        for (int w = 0; w < kWarps; ++w) v.hi += shD[w];
        for (int w = 0; 32 * w < p.numDiag; ++w) v.add(shP[w]);
        partials[blockIdx.x] = v.hi + v.lo;
        __threadfence();
        amLast = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!amLast) return;
    __threadfence();
    acc = 0.0;
    for (unsigned k = tid; k < gridDim.x; k += kThreads) acc += __ldcg(partials + k);
    acc = warpSum(acc);
    if (lane == 0) shD[warp] = acc;
    __syncthreads();
    if (tid == 0) {
        double v = 0;
        for (int w = 0; w < kWarps; ++w) v += shD[w];
        result[0] = v;
        *counter = 0u;
    }
}

// amplitudes, and the qubits of the tile index bits from kLow up
size_t tileShared(int b) { return (size_t(16) << b) + (size_t(8) << (b - kLow)); }

uint32_t localMask(uint64_t mask, const unsigned char* pos, int b) {
    uint32_t l = 0;
    for (int k = 0; k < b; ++k) l |= (uint32_t)(mask >> pos[k] & 1) << k;
    return l;
}

// two terms of one list on one X/Y mask
struct Step {
    uint64_t x, m, d;
    double c[2];
    int imag;
};
struct Plan {
    uint64_t tile = 0;                           // tile qubits, without the forced low ones
    std::vector<Step> steps;
    int first = 0, count = 0;                    // diagonal terms
};

// Steps dealt to passes: each to the pass whose tile grows least for it.
std::vector<Plan> deal(const std::vector<Step>& steps, int numDiag, int b) {
    const int room = b - kLow;
    std::vector<Plan> out;
    for (const Step& s : steps) {
        const uint64_t x = s.x >> kLow << kLow;
        int best = -1, grow = 99;
        for (size_t k = 0; k < out.size(); ++k) {
            const int all = __builtin_popcountll(out[k].tile | x), g = all - __builtin_popcountll(out[k].tile);
            if (all <= room && (int)out[k].steps.size() < kMaxOps && g < grow) {
                best = (int)k;
                grow = g;
            }
        }
        if (best < 0) {
            out.emplace_back();
            best = (int)out.size() - 1;
        }
        out[best].tile |= x;
        out[best].steps.push_back(s);
    }
    for (int d = 0, k = 0; d < numDiag; d += kMaxDiag, ++k) {
        if (k == (int)out.size()) out.emplace_back();
        out[k].first = d;
        out[k].count = std::min(kMaxDiag, numDiag - d);
    }
    return out;
}

}  // namespace

bool expecTileTakes(int n, uint64_t x) {
    return n >= kMinTileBits && __builtin_popcountll(x >> kLow) <= std::min(n, kMaxTileBits) - kLow;
}

bool queueExpecTiles(SV s, const std::vector<PauliTermGroup>& groups, const Scratch& w, const std::function<double*()>& slot,
                     const char* caller) {
    std::vector<Step> steps;
    std::vector<std::pair<uint64_t, double>> diag;
    for (const PauliTermGroup& g : groups) {
        if (g.xmask == 0) {
            for (const PauliTerm& t : g.terms) diag.push_back({t.yz, t.coeff});
            continue;
        }
        std::vector<std::pair<uint64_t, double>> list[2];
        pauliPairTerms(g.xmask, g.terms, list[0], list[1]);
        for (int im = 0; im < 2; ++im)
            for (size_t k = 0; k < list[im].size(); k += 2) {
                Step st{g.xmask, list[im][k].first, 0, {list[im][k].second, 0}, im};
                if (k + 1 < list[im].size()) {
                    st.d = st.m ^ list[im][k + 1].first;
                    st.c[1] = st.c[0] - list[im][k + 1].second;
                    st.c[0] += list[im][k + 1].second;
                }
                if (st.c[0] != 0 || st.c[1] != 0) steps.push_back(st);
            }
    }
    if (steps.empty() && diag.empty()) return true;      // density matrices, small registers: no tile size fits them
    // equal weights next to one another
    std::stable_sort(steps.begin(), steps.end(), [](const Step& a, const Step& b) {
        return a.c[0] != b.c[0] ? a.c[0] < b.c[0] : a.c[1] < b.c[1];
    });
    // tile size: per pass a launch, the state's read, and per SM its tiles'
    // sums; small registers take smaller tiles, so that every SM has one
    int b = 0;
    double best = 0;
    std::vector<Plan> plan;
    const double sms = numSMs();
    for (int c = std::min(s.n, kMinTileBits); c <= std::min(s.n, kMaxTileBits); ++c) {
        bool fits = true;
        for (const Step& st : steps) fits = fits && __builtin_popcountll(st.x >> kLow) <= c - kLow;
        if (!fits) continue;
        std::vector<Plan> p = deal(steps, (int)diag.size(), c);
        double us = 0;
        const double rounds = std::ceil(std::ldexp(1.0, s.n - c) / sms), amps = std::ldexp(1.0, c);
        for (const Plan& q : p) {
            us += 4 + std::ldexp(1.0, s.n) * 16 / 6e6 + rounds * ((q.count ? 3 : 0) + amps * 40 / (90 * 1900));
            for (const Step& a : q.steps)                            // 1.65 FP64 operations a clock
                us += rounds * std::max(0.3, amps * ((a.c[0] == 0) != (a.c[1] == 0) && a.d ? 0.25 : 0.5) * 2 / (1.65 * 1900));
        }
        if (b && us >= best) continue;
        b = c;
        best = us;
        plan.swap(p);
    }
    if (!b) return false;
    cudaStream_t st = stream();
    const size_t smem = tileShared(b);
    if (QG_CUDA(allowShared<kExpecTile>(tileShared(kMaxTileBits)), caller)) return false;
    const uint64_t tiles = 1ull << (s.n - b);
    const unsigned grid = (unsigned)std::min<uint64_t>(tiles, 3ull * (uint64_t)numSMs());
    for (const Plan& pp : plan) {
        ExpecPass p{};
        p.b = b;
        uint64_t tile = pp.tile | ((1ull << kLow) - 1);
        for (int q = 0; q < s.n && __builtin_popcountll(tile) < b; ++q) tile |= 1ull << q;
        for (int q = 0, k = 0; q < s.n; ++q)
            if (tile >> q & 1) p.pos[k++] = (unsigned char)q;
        int run = 0;                             // products in this thread's sum, kept short
        for (size_t i = 0; i < pp.steps.size(); ++i) {
            const Step& a = pp.steps[i];
            PairOp& op = p.op[p.numOps++];
            // without a second term only parity 0 occurs
            op.c[0] = a.c[0];
            op.c[1] = a.d ? a.c[1] : 0;
            op.m = a.m & ~tile;
            op.d = a.d & ~tile;
            op.xl = localMask(a.x, p.pos, b);
            op.ml = localMask(a.m, p.pos, b);
            op.dl = localMask(a.d, p.pos, b);
            op.pair = 31 - __builtin_clz(op.xl);
            op.imag = a.imag;
            const uint32_t free = op.dl & ~(1u << op.pair);
            op.fix = (op.c[0] == 0) != (op.c[1] == 0) && a.d && free ? 31 - __builtin_clz(free) : -1;
            run += 2 * std::max(1, (int)((size_t(1) << (b - 1)) / kThreads));
            const bool more = i + 1 < pp.steps.size();
            const double n1 = more && pp.steps[i + 1].d ? pp.steps[i + 1].c[1] : 0;
            op.flush = !more || pp.steps[i + 1].c[0] != op.c[0] || n1 != op.c[1] || run >= 128;
            if (op.flush) run = 0;
        }
        for (int k = 0; k < pp.count; ++k) {
            p.dm[k] = diag[pp.first + k].first & ~tile;
            p.dml[k] = localMask(diag[pp.first + k].first, p.pos, b);
            p.dc[k] = diag[pp.first + k].second;
        }
        p.numDiag = pp.count;
        double* out = slot();
        if (!out) return false;
        chainShared<kExpecTile>(1, grid, kThreads, smem, st, s.re, s.im, tiles, p, w.partials, w.counter, out);
        if (launchFailed(caller)) return false;
    }
    return true;
}

}  // namespace qg
