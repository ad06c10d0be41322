// reduce.cu -- FP64 reductions in one launch each (sm_103a).
//
// The reference (Code/QuEST340/QuEST/src/GPU/QuEST_gpu.cu:1926-2483) reduces
// level by level with a 512-wide shared-memory tree and a
// cudaDeviceSynchronize per level, runs complex inner products twice (real,
// imaginary), and computes calcTotalProb by copying the whole state to the
// host (:1626-1679).  Here every reduction is a single pass: each thread keeps
// FP64 partial sums of two components, warps combine with
// shuffles, blocks through shared memory, and the last block to finish (a
// ticket counter in the register's scratch) adds the per-block partials in a
// fixed order.  The partial layout depends only on the problem size, so
// results are deterministic run to run.  One scalar pair is copied back.
#include "fixed_sum.cuh"
#include "pauli_expec.h"
#include "reduce_kernel.cuh"

#include <algorithm>
#include <cmath>

namespace qg {
namespace {

using namespace red;

// ------------------------------------------------------------------ functors
// Sums of squares, four amplitudes an item on the integer pipes
// (fixed_sum.cuh).  An item's amplitudes come from `items` apart, so that the
// lanes of a warp read side by side whatever the target.
struct Four {
    double2 a, b, c, d;
};
struct Squares {
    const double *re, *im;
    uint64_t items;
    __device__ __forceinline__ Four pairs(uint64_t i, uint64_t j) const { return Four{ld2(re + i), ld2(re + j), ld2(im + i), ld2(im + j)}; }
    __device__ __forceinline__ double add(double acc, const Four& v) const { return fsum::addSquares(acc, v.a, v.b, v.c, v.d); }
};
struct NormSq4 : Squares {
    __device__ __forceinline__ Four load(uint64_t k) const { return pairs(2 * k, 2 * (k + items)); }
};
struct ProbZero4 : Squares {       // target >= 1: the amplitudes with bit t clear
    int t;
    __device__ __forceinline__ Four load(uint64_t k) const { return pairs(ins0(2 * k, t), ins0(2 * (k + items), t)); }
};
struct ProbZeroEven : Squares {    // target 0
    __device__ __forceinline__ Four load(uint64_t k) const {
        double x[4], y[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            x[u] = ld2(re + 2 * (k + u * items)).x;
            y[u] = ld2(im + 2 * (k + u * items)).x;
        }
        return Four{make_double2(x[0], x[1]), make_double2(x[2], x[3]), make_double2(y[0], y[1]), make_double2(y[2], y[3])};
    }
};
struct NormSq1 {
    const double *re, *im;
    __device__ __forceinline__ double2 operator()(uint64_t i) const {
        const double r = re[i], m = im[i];
        return make_double2(r * r + m * m, 0.0);
    }
};
struct DiagSum {          // sum of Re rho_rr
    const double* re;
    uint64_t step;        // D + 1
    __device__ __forceinline__ double2 operator()(uint64_t r) const { return make_double2(re[r * step], 0.0); }
};
struct ProbZeroFew {      // registers of one or two qubits
    const double *re, *im;
    int t;
    __device__ __forceinline__ double2 operator()(uint64_t k) const {
        const uint64_t i = ins0(k, t);
        return make_double2(re[i] * re[i] + im[i] * im[i], 0.0);
    }
};
struct ProbZeroDiag {     // diagonal entries rho_rr with bit t of r = 0
    const double* re;
    uint64_t step;
    int t;
    __device__ __forceinline__ double2 operator()(uint64_t k) const { return make_double2(re[ins0(k, t) * step], 0.0); }
};
// sum conj(bra) ket, two amplitudes an item on the integer pipes
__device__ __noinline__ double2 innerFp64(double2 a, double2 b, double2 c, double2 d) {
    return make_double2(a.x * c.x + b.x * d.x + a.y * c.y + b.y * d.y, a.x * d.x - b.x * c.x + a.y * d.y - b.y * c.y);
}
struct Inner2 {
    const double *br, *bi, *kr, *ki;
    __device__ __forceinline__ Four load(uint64_t i) const { return Four{ld2(br + 2 * i), ld2(bi + 2 * i), ld2(kr + 2 * i), ld2(ki + 2 * i)}; }
    __device__ __forceinline__ double2 add(double2 acc, const Four& v) const {
        const double2 a = v.a, b = v.b, c = v.c, d = v.d;
        using namespace fsum;
        const uint32_t ma = magnitude(a.x), na = magnitude(a.y), mb = magnitude(b.x), nb = magnitude(b.y);
        const uint32_t mc = magnitude(c.x), nc = magnitude(c.y), md = magnitude(d.x), nd = magnitude(d.y);
        const uint32_t wb = max(max(ma, na), max(mb, nb)), wk = max(max(mc, nc), max(md, nd));
        const int E = (int)(wb >> 20), F = (int)(wk >> 20);
        // (a zero factor adds nothing, unless the other is infinite or NaN)
        if (((wb | lowWords(a, b)) == 0 && F < 0x7FF) || ((wk | lowWords(c, d)) == 0 && E < 0x7FF)) return acc;
        const int ea = exponentOf(ma), eb = exponentOf(mb), ec = exponentOf(mc), ed = exponentOf(md);
        const int fa = exponentOf(na), fb = exponentOf(nb), fc = exponentOf(nc), fd = exponentOf(nd);
        if (!unitFits(E, F) || !productsFit(E, F, ea + ec, eb + ed, fa + fc, fb + fd) ||
            !productsFit(E, F, ea + ed, eb + ec, fa + fd, fb + fc)) {
            const double2 v = innerFp64(a, b, c, d);
            return make_double2(acc.x + v.x, acc.y + v.y);
        }
        const int2 ax = wideDigits(a.x, E), ay = wideDigits(a.y, E), bx = wideDigits(b.x, E), by = wideDigits(b.y, E);
        const int2 cx = wideDigits(c.x, F), cy = wideDigits(c.y, F), dx = wideDigits(d.x, F), dy = wideDigits(d.y, F);
        const int2 nx = make_int2(-bx.x, -bx.y), ny = make_int2(-by.x, -by.y);
        Sums r{0, 0, 0}, m{0, 0, 0};
        r.add(ax, cx); r.add(bx, dx); r.add(ay, cy); r.add(by, dy);
        m.add(ax, dx); m.add(nx, cx); m.add(ay, dy); m.add(ny, cy);
        const double u = wideUnit(E, F);
        return make_double2(fma(u, r.wide(), acc.x), fma(u, m.wide(), acc.y));
    }
};
struct Inner1 {
    const double *br, *bi, *kr, *ki;
    __device__ __forceinline__ double2 operator()(uint64_t i) const {
        return make_double2(br[i] * kr[i] + bi[i] * ki[i], br[i] * ki[i] - bi[i] * kr[i]);
    }
};
struct DistSq {
    const double *ar, *ai, *br, *bi;
    __device__ __forceinline__ double2 operator()(uint64_t i) const {
        const double dr = ar[i] - br[i], di = ai[i] - bi[i];
        return make_double2(dr * dr + di * di, 0.0);
    }
};
// <psi|rho|psi> = sum_{r,c} Re(conj(psi_r) rho_rc psi_c), one entry per item
struct FidelityDM {
    const double *rr, *ri, *pr, *pi;
    int N;
    __device__ __forceinline__ double2 operator()(uint64_t i) const {
        const uint64_t r = i & ((1ull << N) - 1ull), c = i >> N;
        const double er = rr[i], ei = ri[i];
        const double vr = __ldg(pr + c), vi = __ldg(pi + c);
        const double tr = er * vr - ei * vi, ti = er * vi + ei * vr;     // rho_rc psi_c
        const double ur = __ldg(pr + r), ui = -__ldg(pi + r);            // conj(psi_r)
        return make_double2(tr * ur - ti * ui, 0.0);
    }
};

// ---- Pauli-string expectation values -----------------------------------
// GB300 runs FP64 at a small fraction of its FP32 rate, and a Pauli sum
// (C4's 80-term Fermi-Hubbard energy) has many terms per X/Y group, so the
// FP64 work per amplitude, not the read of the state, set the time of these
// reductions.  The per-term algebra is therefore done on the host:
//   * pairs (j, k = j ^ x): with w = conj(psi_j) psi_k and s_q(j) =
//     (-1)^popc(j & yz_q), term q adds c_q s_q(j) [Re((-i)^ph w) +
//     tau_q Re((-i)^ph conj w)], tau_q = (-1)^popc(x & yz_q); that is
//     2 c_q s_q(j) (+-Re w or +-Im w) when tau_q fits the phase, else 0.  An
//     item costs wr A(j) + wi B(j) with A, B = sums of +-c over the terms;
//   * DM, Tr(P rho) = sum_r s(r) Re((-i)^ph rho[r ^ x, r]) = er A(r) + ei B(r);
//   * state vectors of 8 qubits or more go by tiles (expec_tile.cu), except
//     masks of more X/Y qubits than a tile has.
// Reference semantics: QuEST_common.c:506-533 (calcExpecPauliSum: clone,
// apply the Pauli string, inner product, per term).
constexpr int kMaxGroupTerms = 32;
struct PauliPairGroup {          // SV pairs (xmask != 0) or DM entries (any xmask)
    uint64_t xmask;
    int low;                     // lowest bit of xmask (SV)
    int nA, nB;                  // terms on Re w (er), on Im w (ei)
    uint64_t mA[kMaxGroupTerms], mB[kMaxGroupTerms];
    double cA[kMaxGroupTerms], cB[kMaxGroupTerms];
};
// sum_q c_q (-1)^popc(j & m_q) for n >= 1 terms (n - 1 FP64 additions)
__device__ __forceinline__ double signedSum(uint64_t j, const uint64_t* m, const double* c, int n) {
    double a = (__popcll(j & m[0]) & 1) ? -c[0] : c[0];
    for (int q = 1; q < n; ++q) a += (__popcll(j & m[q]) & 1) ? -c[q] : c[q];
    return a;
}

// x A(j) + y B(j) for a group with at least one term, skipping an empty list
// (the counts are uniform across the launch)
__device__ __forceinline__ double pairValue(uint64_t j, double x, double y, const PauliPairGroup& g) {
    if (g.nB == 0) return x * signedSum(j, g.mA, g.cA, g.nA);
    if (g.nA == 0) return y * signedSum(j, g.mB, g.cB, g.nB);
    return fma(x, signedSum(j, g.mA, g.cA, g.nA), y * signedSum(j, g.mB, g.cB, g.nB));
}
struct ExpecPairs {
    const double *re, *im;
    PauliPairGroup g;
    __device__ __forceinline__ double2 operator()(uint64_t t) const {
        const uint64_t j = ins0(t, g.low), k = j ^ g.xmask;
        const double jr = re[j], ji = im[j], kr = re[k], ki = im[k];
        // conj(psi_j) psi_k, only the parts the group's terms use
        const double wr = g.nA ? fma(jr, kr, ji * ki) : 0.0;
        const double wi = g.nB ? fma(jr, ki, -(ji * kr)) : 0.0;
        return make_double2(pairValue(j, wr, wi, g), 0.0);
    }
};
struct ExpecDM {
    const double *re, *im;
    PauliPairGroup g;
    int N;
    __device__ __forceinline__ double2 operator()(uint64_t r) const {
        const uint64_t idx = (r ^ g.xmask) + (r << N);
        return make_double2(pairValue(r, re[idx], im[idx], g), 0.0);
    }
};
struct ExpecDiag1 {                              // SV, x = 0, one amplitude per item (n < 8)
    const double *re, *im;
    PauliPairGroup g;
    __device__ __forceinline__ double2 operator()(uint64_t j) const {
        return make_double2(pairValue(j, re[j] * re[j] + im[j] * im[j], 0.0, g), 0.0);
    }
};

// ---- calcProbOfAllOutcomes ------------------------------------------------
// The amplitude index is the low qubits, one value per thread of a unit, and
// the rest, the items: (values of the measured high qubits, values of the
// others), the others fastest.  A unit takes a run of items; a thread sums its
// amplitudes while the measured high qubits stay, four at a time on the
// integer pipes, and the unit then adds its threads of equal outcome and gives
// the sums to out.  A unit is a block (8 low qubits); where a block's runs
// would be short (most high qubits measured) and its adding, five FP64
// additions by every thread a run, all the work, it is a warp (5 low qubits).
// 24 qubits (HBM floor 39 us), 10 measured: 119 us with an atomic addition per
// amplitude, 46 so; 16 measured, the highest (the whole call, with its copy to
// the host): 270, by blocks 507, by warps 130.
constexpr int kLowQubits = 8, kWarpQubits = 5;
struct OutcomeSpec {
    unsigned char low, high;            // low qubits (kLowQubits or kWarpQubits, or all of fewer), the other ones
    unsigned char numMeasured;          // high qubits that are measured
    unsigned char lowMask;              // low qubits that are measured
    unsigned char lowBit[kLowQubits];   // the outcome's bit of each low qubit
    uint64_t measured;                  // the measured high qubits (bit 0: qubit `low`)
    unsigned char highQubit[40];        // ascending, likewise
    unsigned char highBit[40];          // the outcome's bit of each
};
template <bool DM, bool WARPS>
__global__ void __launch_bounds__(1 << kLowQubits) kOutcomes(const double* __restrict__ re, const double* __restrict__ im,
                                                             uint64_t step, const __grid_constant__ OutcomeSpec s,
                                                             double* __restrict__ out) {
    constexpr int kUnitQubits = WARPS ? kWarpQubits : kLowQubits, kPerBlock = 1 << (kLowQubits - kUnitQubits);
    __shared__ double part[1 << kLowQubits];
    const uint32_t tid = threadIdx.x & ((1u << kUnitQubits) - 1u);
    const bool live = tid < 1u << s.low;
    const uint64_t others = ((1ull << s.high) - 1) & ~s.measured;
    const int fast = s.high - s.numMeasured;
    const uint64_t items = 1ull << s.high;
    const uint64_t unit = (uint64_t)blockIdx.x * kPerBlock + (threadIdx.x >> kUnitQubits), units = (uint64_t)gridDim.x * kPerBlock;
    const uint64_t each = items / units, more = items % units;
    uint64_t k = each * unit + min(unit, more);
    const uint64_t end = k + each + (unit < more ? 1 : 0);
    // the first item's qubits and outcome
    uint64_t set = 0, h = 0, v = k >> fast, r = k & ((1ull << fast) - 1);
    uint32_t o = 0;
    for (int q = 0; q < s.low; ++q)
        if (s.lowMask >> q & 1u) o |= ((tid >> q) & 1u) << s.lowBit[q];
    for (int m = 0; m < s.numMeasured; ++m) {
        const uint32_t bit = (uint32_t)(v >> m) & 1u;
        set |= (uint64_t)bit << s.highQubit[m];
        o |= bit << s.highBit[m];
    }
    for (int q = 0; r; ++q) {
        if (s.measured >> q & 1) continue;
        h |= (r & 1) << q;
        r >>= 1;
    }
    while (k < end) {
        // a run with the same measured high qubits
        const uint64_t stop = min(end, ((k >> fast) + 1) << fast);
        double acc = 0.0;
        for (; k < stop; k += 4) {
            double x[4] = {0, 0, 0, 0}, y[4] = {0, 0, 0, 0};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (live && k + u < stop) {
                    const uint64_t i = (((set | h) << s.low) | tid) * step;
                    x[u] = re[i];
                    if (!DM) y[u] = im[i];
                }
                h = ((h | ~others) + 1) & others;
            }
            if (DM) acc += (x[0] + x[1]) + (x[2] + x[3]);
            else if (stop - k == 1) acc = fma(x[0], x[0], fma(y[0], y[0], acc));        // one amplitude: FP64 is less work
            else acc = fsum::addSquares(acc, make_double2(x[0], x[1]), make_double2(x[2], x[3]), make_double2(y[0], y[1]), make_double2(y[2], y[3]));
        }
        k = stop;
        h = 0;
        // the threads that differ in unmeasured low qubits only (those that a
        // small register lacks too): lanes, then warps
        const uint32_t skip = ~(uint32_t)s.lowMask & ((1u << kUnitQubits) - 1u);
#pragma unroll
        for (int q = 0; q < 5; ++q)
            if (skip >> q & 1u) acc += __shfl_xor_sync(0xffffffffu, acc, 1 << q);
        if (!WARPS && skip >> 5) {
            __syncthreads();
            part[tid] = acc;
            __syncthreads();
            for (uint32_t w = 1; w < 8; ++w)
                if (((w << 5) & ~skip) == 0 && (tid & skip) == 0) acc += part[tid | (w << 5)];
        }
        if ((tid & skip) == 0) atomicAdd(out + o, acc);
        uint64_t changed = v ^ (v + 1);          // the next run's measured qubits
        ++v;
        for (int m = 0; changed && m < s.numMeasured; ++m, changed >>= 1) {
            set ^= 1ull << s.highQubit[m];
            o ^= 1u << s.highBit[m];
        }
    }
}

}  // namespace

// ============================================================== public API
double reduceTotalProbSV(SV s, const Scratch& w) {                 // replaces QuEST_gpu.cu:1649-1679
    double v = 0;
    const uint64_t n = 1ull << s.n;
    if (n >= 4) runSum<double>(NormSq4{{s.re, s.im, n / 4}}, n / 4, w, &v, nullptr, "calcTotalProb");
    else runReduce(NormSq1{s.re, s.im}, n, w, &v, nullptr, "calcTotalProb");
    return v;
}

double reduceNormSq(SV s, const Scratch& w) { return reduceTotalProbSV(s, w); }

double reduceTotalProbDM(SV s, int N, const Scratch& w) {          // replaces QuEST_gpu.cu:1626-1647
    double v = 0;
    runReduce(DiagSum{s.re, (1ull << N) + 1}, 1ull << N, w, &v, nullptr, "calcTotalProb");
    return v;
}

double reduceProbZeroSV(SV s, int t, const Scratch& w) {           // QuEST_gpu.cu:1992-2161
    double v = 0;
    const uint64_t half = 1ull << (s.n - 1);
    if (half < 4) runReduce(ProbZeroFew{s.re, s.im, t}, half, w, &v, nullptr, "calcProbOfOutcome");
    else if (t >= 1) runSum<double>(ProbZero4{{s.re, s.im, half / 4}, t}, half / 4, w, &v, nullptr, "calcProbOfOutcome");
    else runSum<double>(ProbZeroEven{{s.re, s.im, half / 4}}, half / 4, w, &v, nullptr, "calcProbOfOutcome");
    return v;
}

double reduceProbZeroDM(SV s, int t, int N, const Scratch& w) {    // QuEST_gpu.cu:1954-2104
    double v = 0;
    runReduce(ProbZeroDiag{s.re, (1ull << N) + 1, t}, 1ull << (N - 1), w, &v, nullptr, "calcProbOfOutcome");
    return v;
}

void reduceInnerProduct(SV bra, SV ket, const Scratch& w, double* outRe, double* outIm) {   // QuEST_gpu.cu:2368-2483
    const uint64_t n = 1ull << bra.n;
    if (n >= 2) runSum<double2>(Inner2{bra.re, bra.im, ket.re, ket.im}, n / 2, w, outRe, outIm, "calcInnerProduct");
    else runReduce(Inner1{bra.re, bra.im, ket.re, ket.im}, n, w, outRe, outIm, "calcInnerProduct");
}

double reduceDotReal(SV a, SV b, const Scratch& w) {               // QuEST_gpu.cu:2297-2366
    double re = 0;
    reduceInnerProduct(a, b, w, &re, nullptr);
    return re;
}

double reduceDistSq(SV a, SV b, const Scratch& w) {
    double v = 0;
    runReduce(DistSq{a.re, a.im, b.re, b.im}, 1ull << a.n, w, &v, nullptr, "calcHilbertSchmidtDistance");
    return v;
}

double reduceFidelityDM(SV rho, SV psi, int N, const Scratch& w) { // replaces QuEST_gpu.cu:2486-2572
    double v = 0;
    runReduce(FidelityDM{rho.re, rho.im, psi.re, psi.im, N}, 1ull << rho.n, w, &v, nullptr, "calcFidelity");
    return v;
}

void pauliPairTerms(uint64_t x, const std::vector<PauliTerm>& terms, std::vector<std::pair<uint64_t, double>>& A,
                    std::vector<std::pair<uint64_t, double>>& B) {
    for (const PauliTerm& t : terms) {
        const int ph = t.nY & 3;
        const bool tauPlus = (__builtin_popcountll(x & t.yz) & 1) == 0;
        if (ph % 2 == 0 && tauPlus) A.push_back({t.yz, ph == 0 ? 2 * t.coeff : -2 * t.coeff});
        if (ph % 2 == 1 && !tauPlus) B.push_back({t.yz, ph == 1 ? 2 * t.coeff : -2 * t.coeff});
    }
}

double reduceExpecPauliGroups(SV s, int isDM, int N, const std::vector<PauliTermGroup>& groups, const Scratch& w) {
    // Every group (or chunk of a large group) reduces into its own result
    // slot; the slots are read back once per 32 launches, and summed on the
    // host in group order.
    constexpr int kSlots = 32;                   // the scratch holds 64 result doubles
    const char* caller = "calcExpecPauliSum";
    cudaStream_t st = stream();
    double total = 0.0, low = 0.0;
    int used = 0;
    auto drain = [&]() -> bool {
        if (!used) return true;
        if (QG_CUDA(cudaMemcpyAsync(w.host, w.result, 2 * used * sizeof(double), cudaMemcpyDeviceToHost, st), caller) ||
            QG_CUDA(cudaStreamSynchronize(st), caller))
            return false;
        for (int k = 0; k < used; ++k) {         // (TwoSum)
            const double x = w.host[2 * k], s = total + x, z = s - total;
            low += (total - (s - z)) + (x - z);
            total = s;
        }
        used = 0;
        return true;
    };
    auto queue = [&](auto f, uint64_t nItems) -> bool {
        if (used == kSlots && !drain()) return false;
        const int grid = reduceGrid(nItems);
        kReduce<<<grid, red::kThreads, 0, st>>>(f, nItems, w.partials, w.counter, w.result + 2 * used);
        if (launchFailed(caller)) return false;
        ++used;
        return true;
    };
    // state vectors go by tiles, except masks wider than a tile
    std::vector<PauliTermGroup> tiled, rest;
    for (const PauliTermGroup& grp : groups) (!isDM && expecTileTakes(s.n, grp.xmask) ? tiled : rest).push_back(grp);
    const bool queued = queueExpecTiles(s, tiled, w, [&]() -> double* {
        if (used == kSlots && !drain()) return nullptr;
        return w.result + 2 * used++;
    }, caller);
    if (!queued) return total;
    for (const PauliTermGroup& grp : rest) {
        const uint64_t x = grp.xmask;
        // pairs / DM entries: each term goes to the Re (A) or Im (B) list
        std::vector<std::pair<uint64_t, double>> A, B;
        if (isDM) {
            for (const PauliTerm& t : grp.terms) {
                const int ph = t.nY & 3;
                (ph % 2 == 0 ? A : B).push_back({t.yz, ph < 2 ? t.coeff : -t.coeff});
            }
        } else if (x == 0) {                     // n < 8 diagonal group: |psi_j|^2 terms
            for (const PauliTerm& t : grp.terms) A.push_back({t.yz, t.coeff});
        } else {
            pauliPairTerms(x, grp.terms, A, B);
        }
        for (size_t a0 = 0, b0 = 0; a0 < A.size() || b0 < B.size();) {
            PauliPairGroup g{};
            g.xmask = x;
            g.low = x ? __builtin_ctzll(x) : 0;
            for (; a0 < A.size() && g.nA < kMaxGroupTerms; ++a0, ++g.nA) {
                g.mA[g.nA] = A[a0].first;
                g.cA[g.nA] = A[a0].second;
            }
            for (; b0 < B.size() && g.nB < kMaxGroupTerms; ++b0, ++g.nB) {
                g.mB[g.nB] = B[b0].first;
                g.cB[g.nB] = B[b0].second;
            }
            bool ok;
            if (isDM) ok = queue(ExpecDM{s.re, s.im, g, N}, 1ull << N);
            else if (x) ok = queue(ExpecPairs{s.re, s.im, g}, 1ull << (s.n - 1));
            else ok = queue(ExpecDiag1{s.re, s.im, g}, 1ull << s.n);
            if (!ok) return total;
        }
    }
    drain();
    return std::isfinite(total) ? total + low : total;
}

void reduceProbAllOutcomes(SV s, int isDM, int N, const int* qubits, int nq, double* hostOut, const Scratch& w) {
    (void)w;
    const int nOut = 1 << nq;
    const size_t bytes = (size_t)nOut * sizeof(double);
    static double* dOut = nullptr;
    static size_t cap = 0;
    if (bytes > cap) {
        if (dOut) cudaFree(dOut);
        dOut = nullptr;
        cap = 0;
        if (QG_CUDA(cudaMalloc(&dOut, bytes), "calcProbOfAllOutcomes")) return;
        cap = bytes;
    }
    cudaStream_t st = stream();
    if (QG_CUDA(cudaMemsetAsync(dOut, 0, (size_t)nOut * sizeof(double), st), "calcProbOfAllOutcomes")) return;
    const int n = isDM ? N : s.n;
    auto spec = [&](int lowest) {
        OutcomeSpec sp{};
        sp.low = (unsigned char)std::min(n, lowest);
        sp.high = (unsigned char)(n - sp.low);
        for (int q = 0; q < n; ++q)
            for (int b = 0; b < nq; ++b) {
                if (qubits[b] != q) continue;
                if (q < sp.low) {
                    sp.lowMask |= 1u << q;
                    sp.lowBit[q] = (unsigned char)b;
                } else {
                    sp.measured |= 1ull << (q - sp.low);
                    sp.highQubit[sp.numMeasured] = (unsigned char)(q - sp.low);
                    sp.highBit[sp.numMeasured++] = (unsigned char)b;
                }
            }
        return sp;
    };
    OutcomeSpec sp = spec(kLowQubits);
    const bool warps = sp.numMeasured > 0 && sp.high - sp.numMeasured < 4;       // runs of fewer than 16 items
    if (warps) sp = spec(kWarpQubits);
    const uint64_t blocks = warps ? ((1ull << sp.high) + 7) / 8 : 1ull << sp.high;
    const unsigned grid = (unsigned)std::min<uint64_t>(blocks, 8ull * (uint64_t)numSMs());
    const uint64_t step = isDM ? (1ull << N) + 1 : 1;
    if (isDM && warps) kOutcomes<true, true><<<grid, 1 << kLowQubits, 0, st>>>(s.re, s.im, step, sp, dOut);
    else if (isDM) kOutcomes<true, false><<<grid, 1 << kLowQubits, 0, st>>>(s.re, s.im, step, sp, dOut);
    else if (warps) kOutcomes<false, true><<<grid, 1 << kLowQubits, 0, st>>>(s.re, s.im, step, sp, dOut);
    else kOutcomes<false, false><<<grid, 1 << kLowQubits, 0, st>>>(s.re, s.im, step, sp, dOut);
    if (launchFailed("calcProbOfAllOutcomes")) return;
    QG_CUDA(cudaMemcpyAsync(hostOut, dOut, (size_t)nOut * sizeof(double), cudaMemcpyDeviceToHost, st), "calcProbOfAllOutcomes");
    QG_CUDA(cudaStreamSynchronize(st), "calcProbOfAllOutcomes");
}

}  // namespace qg
