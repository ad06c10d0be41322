// sv_gates.cu -- plain FP64 gate kernels for sm_103a.
//
// One launch per API gate, each a single streaming pass over only the
// amplitudes the gate touches (control bits are enumerated, not tested), with
// 16-byte vector loads of the SoA real/imag arrays.  Semantics follow the
// reference backend Code/QuEST340/QuEST/src/GPU/QuEST_gpu.cu (line numbers
// per launcher below); the thread->amplitude mapping is new.
//
// Thread mapping.  A gate touches pairs (i0, i0 ^ pmask) whose "inserted"
// bits (the lowest partner bit plus all control bits) are fixed: i0 =
// insertZeros(k) | setMask for k in [0, 2^(n - numInserted)).  When no
// inserted bit is bit 0, consecutive k give consecutive i0, so one thread
// takes k = 2t, 2t+1 and moves them with double2 loads (kVec).  When the
// partner bit is bit 0 the pair itself is adjacent (kAdj).  Otherwise kScalar.
#include "chain_launch.cuh"
#include "df64.cuh"
#include "fix64.cuh"
#include "qg_internal.h"

#include <algorithm>
#include <vector>

namespace qg {

namespace {

constexpr int kThreads = 256;

struct InsSpec {
    int n;
    int pos[63];   // ascending bit positions of the zeros to insert
};

__device__ __forceinline__ uint64_t insertZeros(uint64_t k, const InsSpec& s) {
    for (int j = 0; j < s.n; ++j) {
        const int b = s.pos[j];
        const uint64_t lo = k & ((1ull << b) - 1ull);
        k = ((k >> b) << (b + 1)) | lo;
    }
    return k;
}

InsSpec makeIns(uint64_t mask) {
    InsSpec s{};
    s.n = 0;
    for (int b = 0; b < 64; ++b)
        if (mask >> b & 1ull) s.pos[s.n++] = b;
    return s;
}

inline unsigned blocksFor(uint64_t threads) { return (unsigned)((threads + kThreads - 1) / kThreads); }

__device__ __forceinline__ double2 ld2(const double* p) { return *reinterpret_cast<const double2*>(p); }
__device__ __forceinline__ void st2(double* p, double2 v) { *reinterpret_cast<double2*>(p) = v; }

// ---------------------------------------------------------------- pair ops
struct OpMatrix2 {
    Mat2 m;
    __device__ __forceinline__ void operator()(double& ur, double& ui, double& lr, double& li) const {
        const double a = ur, b = ui, c = lr, d = li;
        ur = m.r[0][0] * a - m.i[0][0] * b + m.r[0][1] * c - m.i[0][1] * d;
        ui = m.r[0][0] * b + m.i[0][0] * a + m.r[0][1] * d + m.i[0][1] * c;
        lr = m.r[1][0] * a - m.i[1][0] * b + m.r[1][1] * c - m.i[1][1] * d;
        li = m.r[1][0] * b + m.i[1][0] * a + m.r[1][1] * d + m.i[1][1] * c;
    }
};

// The same update in fixed point on the integer pipes (fix64.cuh): the four
// reals of a pair under the matrix's real 4 x 4 form.  Pairs whose exponents
// are out of its range (all zero, among others) take the FP64 arithmetic,
// (OpFixed2: behind a call: inlined, its few FP64 instructions would be predicated, and
// a predicated-off instruction still takes its slots of the FP64 pipe).
//
// With all warps in fixed point the FP64 pipe (whose conversions end each
// output) is half idle while the integer pipes bound the kernel, so one warp
// in kFp64Share works in FP64.  One gate at 26 qubits (targets 0, 3, 25):
// all in FP64 1024 us, all in fixed point 430, 414, 425; shared at 1 in 7
// 407, 387, 397 (6: 404, 384, 391; 10: 429, 400, 412).  HBM floor 316; at 20
// qubits 20 us before, 10.3 now.  A warp of 1 in 7 takes turns on the SM's
// partitions, as a power of two would not.
constexpr unsigned kFp64Share = 7;
__device__ __noinline__ double2 real2Rare(double a, double b, double c, double d, double x, double y) {
    return make_double2(a * x + b * y, c * x + d * y);
}
struct OpFixed4 {
    fx::Map<4> f;
    OpMatrix2 exact;
    __device__ __forceinline__ void operator()(double& ur, double& ui, double& lr, double& li) const {
        double* const x[4] = {&ur, &ui, &lr, &li};
        const unsigned warp = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
        if (warp % kFp64Share == 0 || !fx::apply<4>(f, x)) exact(ur, ui, lr, li);
    }
};
// A matrix whose real form couples ur only with lr and ui only with li (a
// real matrix) or, after lr and li change places (launchPair's `cross`), ur
// only with li and ui only with lr (rotateX): two real 2 x 2 maps, half the
// products of the general form.  rotateY at 26 qubits: 1024 us in the general
// FP64 form, 330, 321, 332 in fixed point (HBM-bound); the same two maps in
// FP64, for matrices that do not fit, take half the general form's time.
struct OpDirect2 {
    double a[2][2], b[2][2];
    __device__ __forceinline__ void operator()(double& ur, double& ui, double& lr, double& li) const {
        const double x = ur, y = ui;
        ur = a[0][0] * x + a[0][1] * lr;
        lr = a[1][0] * x + a[1][1] * lr;
        ui = b[0][0] * y + b[0][1] * li;
        li = b[1][0] * y + b[1][1] * li;
    }
};
__device__ __forceinline__ void fixed2(const fx::Map<2>& f, const double (&m)[2][2], double& x, double& y) {
    double* const p[2] = {&x, &y};
    if (!fx::apply<2>(f, p)) {
        const double2 v = real2Rare(m[0][0], m[0][1], m[1][0], m[1][1], x, y);
        x = v.x;
        y = v.y;
    }
}
struct OpFixed2 {
    fx::Map<2> fa, fb;
    OpDirect2 exact;
    __device__ __forceinline__ void operator()(double& ur, double& ui, double& lr, double& li) const {
        fixed2(fa, exact.a, ur, lr);
        fixed2(fb, exact.b, ui, li);
    }
};

// The 2 x 2 update in double-float form (df64.cuh), for the plain path's
// double-float mode (quest_gb300_setPlainArithmetic(1)): each output is a
// compensated four-term dot product of DF coefficients and the DF parts of
// the inputs, on the FP32 and integer pipes.  coef[o] holds the four
// coefficients of output o (ur, ui, lr, li) against inputs (a, b, c, d) =
// (ur, ui, lr, li) for the real outputs and (b, a, d, c) for the imaginary
// ones, signs included.
struct OpMatrix2DF {
    df::F2 coef[4][4];
    __device__ __forceinline__ void operator()(double& ur, double& ui, double& lr, double& li) const {
        const df::F2 a = df::fromDouble(ur), b = df::fromDouble(ui), c = df::fromDouble(lr), d = df::fromDouble(li);
        const df::F2 re4[4] = {a, b, c, d}, im4[4] = {b, a, d, c};
        ur = df::toDouble(df::dot4(coef[0], re4));
        ui = df::toDouble(df::dot4(coef[1], im4));
        lr = df::toDouble(df::dot4(coef[2], re4));
        li = df::toDouble(df::dot4(coef[3], im4));
    }
};
OpMatrix2DF matrix2DF(const Mat2& m) {
    OpMatrix2DF op;
    const double k[4][4] = {{m.r[0][0], -m.i[0][0], m.r[0][1], -m.i[0][1]},
                            {m.r[0][0], m.i[0][0], m.r[0][1], m.i[0][1]},
                            {m.r[1][0], -m.i[1][0], m.r[1][1], -m.i[1][1]},
                            {m.r[1][0], m.i[1][0], m.r[1][1], m.i[1][1]}};
    for (int o = 0; o < 4; ++o)
        for (int j = 0; j < 4; ++j) op.coef[o][j] = df::splitConst(k[o][j]);
    return op;
}
// 0: FP64 and fixed point at its precision (the default); 1: double-float for the general 2 x 2 gates
int g_plainArith = 0;

struct OpSwap {
    __device__ __forceinline__ void operator()(double& ur, double& ui, double& lr, double& li) const {
        double t = ur; ur = lr; lr = t;
        t = ui; ui = li; li = t;
    }
};

// QuEST_gpu.cu:1362-1455: up' = c*(im_lo, -re_lo), lo' = c*(-im_up, re_up)
struct OpPauliY {
    double c;
    __device__ __forceinline__ void operator()(double& ur, double& ui, double& lr, double& li) const {
        const double a = ur, b = ui, x = lr, y = li;
        ur = c * y; ui = -c * x;
        lr = -c * b; li = c * a;
    }
};

// lre, lim: the arrays of the partner's parts; the same as re and im, or im
// and re when the op couples ur with li and ui with lr (`cross`)
template <class Op>
__global__ void __launch_bounds__(kThreads, 6) kPairVec(double* re, double* im, double* lre, double* lim, InsSpec ins,
                                                     uint64_t setMask, uint64_t pmask, uint64_t nThreads, Op op) {
    const uint64_t t = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
    if (t >= nThreads) return;
    const uint64_t i0 = insertZeros(t << 1, ins) | setMask;
    const uint64_t i1 = i0 ^ pmask;
    chainStart();
    double2 ur = ld2(re + i0), ui = ld2(im + i0), lr = ld2(lre + i1), li = ld2(lim + i1);
    op(ur.x, ui.x, lr.x, li.x);
    op(ur.y, ui.y, lr.y, li.y);
    st2(re + i0, ur); st2(im + i0, ui); st2(lre + i1, lr); st2(lim + i1, li);
}

// partner bit is bit 0: (re[i0], re[i0+1]) is one pair; two pairs per thread
template <bool CROSS, class Op>
__global__ void __launch_bounds__(kThreads) kPairAdj(double* re, double* im, InsSpec ins,
                                                     uint64_t setMask, uint64_t nThreads, Op op) {
    const uint64_t t = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
    if (t >= nThreads) return;
    const uint64_t a0 = insertZeros(t << 1, ins) | setMask;
    const uint64_t a1 = insertZeros((t << 1) | 1ull, ins) | setMask;
    chainStart();
    double2 r0 = ld2(re + a0), i0 = ld2(im + a0), r1 = ld2(re + a1), i1 = ld2(im + a1);
    op(r0.x, i0.x, CROSS ? i0.y : r0.y, CROSS ? r0.y : i0.y);
    op(r1.x, i1.x, CROSS ? i1.y : r1.y, CROSS ? r1.y : i1.y);
    st2(re + a0, r0); st2(im + a0, i0); st2(re + a1, r1); st2(im + a1, i1);
}

template <class Op>
__global__ void __launch_bounds__(kThreads) kPairScalar(double* re, double* im, double* lre, double* lim, InsSpec ins,
                                                        uint64_t setMask, uint64_t pmask, uint64_t nPairs, Op op) {
    const uint64_t t = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
    if (t >= nPairs) return;
    const uint64_t i0 = insertZeros(t, ins) | setMask;
    const uint64_t i1 = i0 ^ pmask;
    chainStart();
    double ur = re[i0], ui = im[i0], lr = lre[i1], li = lim[i1];
    op(ur, ui, lr, li);
    re[i0] = ur; im[i0] = ui; lre[i1] = lr; lim[i1] = li;
}

// Launch a pair gate: partner = i0 ^ pmask, lowBit = lowest bit of pmask
// (inserted as 0 in i0), ctrl bits inserted and set according to setMask.
template <class Op>
void launchPair(SV s, uint64_t ctrl, uint64_t setMask, uint64_t pmask, const Op& op, const char* caller, bool cross = false) {
    const uint64_t lowBit = pmask & (~pmask + 1ull);
    const uint64_t insMask = ctrl | lowBit;
    const InsSpec ins = makeIns(insMask);
    const int free = s.n - ins.n;
    if (free < 0) return;
    const uint64_t nPairs = 1ull << free;
    cudaStream_t st = stream();
    double* const lre = cross ? s.im : s.re;
    double* const lim = cross ? s.re : s.im;
    if (nPairs >= 2 && !(insMask & 1ull)) {
        chain<kPairVec<Op>>(blocksFor(nPairs / 2), kThreads, st, s.re, s.im, lre, lim, ins, setMask, pmask, nPairs / 2, op);
    } else if (nPairs >= 2 && pmask == 1ull) {
        if (cross) chain<kPairAdj<true, Op>>(blocksFor(nPairs / 2), kThreads, st, s.re, s.im, ins, setMask, nPairs / 2, op);
        else chain<kPairAdj<false, Op>>(blocksFor(nPairs / 2), kThreads, st, s.re, s.im, ins, setMask, nPairs / 2, op);
    } else {
        chain<kPairScalar<Op>>(blocksFor(nPairs), kThreads, st, s.re, s.im, lre, lim, ins, setMask, pmask, nPairs, op);
    }
    launchFailed(caller);
}

// ------------------------------------------------------- elementwise (diagonal)
// An op is told the parity of idx & targ, which is linear in idx: a kernel
// works it out once for amplitudes idx, idx + 1.
struct OpPhase {           // amp *= t
    double tr, ti;
    __device__ __forceinline__ int odd(uint64_t) const { return 0; }
    __device__ __forceinline__ void operator()(int, double& r, double& i) const {
        const double a = r, b = i;
        r = tr * a - ti * b;
        i = ti * a + tr * b;
    }
};

// QuEST_gpu.cu:1565-1591: even parity -> exp(-i a/2), odd -> exp(+i a/2)
struct OpRotZ {
    uint64_t targ;
    double c, s;
    __device__ __forceinline__ int odd(uint64_t idx) const { return __popcll(idx & targ) & 1; }
    __device__ __forceinline__ void operator()(int one, double& r, double& i) const {
        const double fs = one ? 1.0 : -1.0;
        const double a = r, b = i;
        r = c * a - fs * s * b;
        i = fs * s * a + c * b;
    }
};

// diag(a, d) on a qubit
struct OpDiag2 {
    uint64_t targ;
    double ar, ai, dr, di;
    __device__ __forceinline__ int odd(uint64_t idx) const { return (idx & targ) != 0; }
    __device__ __forceinline__ void operator()(int one, double& r, double& i) const {
        const double tr = one ? dr : ar, ti = one ? di : ai, x = r, y = i;
        r = tr * x - ti * y;
        i = ti * x + tr * y;
    }
};

// OpRotZ in fixed point (fix64.cuh): [c s; -s c] on (re, im), its inverse for
// odd parity (the map between two changes of the imaginary part's sign).  Four
// FP64 operations an amplitude leave HBM half idle; the fixed-point map has
// two (the conversions at its end), but keeps the integer pipes 76 % busy, so
// one warp in kTurnFp64Share works in FP64.  rotateZ at 26 qubits (HBM floor
// 316 us): as a general matrix 1023 us, all in fixed point 362, one warp in 3,
// 4, 5, 7 in FP64 330, 317, 334, 346.  phaseShift there (floor 158) 203 all in
// fixed point, 168 so; controlledPhaseShift on a quarter of the amplitudes
// (floor 79) 133 in FP64, 107-121.
constexpr unsigned kTurnFp64Share = 4;
struct OpTurnFixed {
    uint64_t targ;
    fx::Map<2> f;
    double m[2][2];
    __device__ __forceinline__ int odd(uint64_t idx) const { return __popcll(idx & targ) & 1; }
    __device__ __forceinline__ void operator()(int one, double& r, double& i) const {
        const int sign = one << 31;
        double v = __hiloint2double(__double2hiint(i) ^ sign, __double2loint(i));
        const unsigned warp = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
        double* const x[2] = {&r, &v};
        if (warp % kTurnFp64Share == 0 || !fx::apply<2>(f, x)) {
            const double2 w = real2Rare(m[0][0], m[0][1], m[1][0], m[1][1], r, v);
            r = w.x;
            v = w.y;
        }
        i = __hiloint2double(__double2hiint(v) ^ sign, __double2loint(v));
    }
};

template <class Op>
__global__ void __launch_bounds__(kThreads) kDiagVec(double* re, double* im, InsSpec ins,
                                                     uint64_t setMask, uint64_t nThreads, Op op) {
    const uint64_t t = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
    if (t >= nThreads) return;
    const uint64_t i0 = insertZeros(t << 1, ins) | setMask;
    chainStart();
    double2 r = ld2(re + i0), m = ld2(im + i0);
    const int one = op.odd(i0);
    op(one, r.x, m.x);
    op(one ^ op.odd(1), r.y, m.y);
    st2(re + i0, r); st2(im + i0, m);
}

template <class Op>
__global__ void __launch_bounds__(kThreads) kDiagScalar(double* re, double* im, InsSpec ins,
                                                        uint64_t setMask, uint64_t nAmps, Op op) {
    const uint64_t t = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
    if (t >= nAmps) return;
    const uint64_t i = insertZeros(t, ins) | setMask;
    chainStart();
    double r = re[i], m = im[i];
    op(op.odd(i), r, m);
    re[i] = r; im[i] = m;
}

template <class Op>
void launchDiag(SV s, uint64_t fixedMask, uint64_t setMask, const Op& op, const char* caller) {
    const InsSpec ins = makeIns(fixedMask);
    const int free = s.n - ins.n;
    if (free < 0) return;
    const uint64_t nAmps = 1ull << free;
    cudaStream_t st = stream();
    if (nAmps >= 2 && !(fixedMask & 1ull))
        chain<kDiagVec<Op>>(blocksFor(nAmps / 2), kThreads, st, s.re, s.im, ins, setMask, nAmps / 2, op);
    else
        chain<kDiagScalar<Op>>(blocksFor(nAmps), kThreads, st, s.re, s.im, ins, setMask, nAmps, op);
    launchFailed(caller);
}

// amp *= c - i s where idx & targ has even parity, c + i s where it has odd:
// in fixed point unless c or s is small, else in FP64
template <class Op>
void launchTurn(SV s, uint64_t fixedMask, uint64_t setMask, uint64_t targ, double c, double sn, const Op& exact, const char* caller) {
    OpTurnFixed f{targ, {}, {{c, sn}, {-sn, c}}};
    if (fx::mapFits<2>(f.m, f.f)) launchDiag(s, fixedMask, setMask, f, caller);
    else launchDiag(s, fixedMask, setMask, exact, caller);
}

// ------------------------------------------------------- Pauli-string rotation
// exp(-i a/2 P) in one pass over pairs (j, j^x).  (P psi)[j] =
// (-i)^nY (-1)^popc(j & (y|z)) psi[j^x]; new[j] = c psi[j] + s g sgn_j psi[j^x]
// with g = -i (-i)^nY (conj: conj(g)).  Replaces the basis-change sequence of
// QuEST_common.c:411-448 (2*#XY + 1 passes) by one pass.
struct PauliRot {
    uint64_t xmask, yz;
    double c, s, gr, gi;
};

__device__ __forceinline__ void pauliPair(const PauliRot& p, uint64_t j, double& jr, double& ji, double& kr, double& ki) {
    const uint64_t k = j ^ p.xmask;
    const double sj = (__popcll(j & p.yz) & 1) ? -p.s : p.s;
    const double sk = (__popcll(k & p.yz) & 1) ? -p.s : p.s;
    const double ar = jr, ai = ji, br = kr, bi = ki;
    // g*b
    const double gbr = p.gr * br - p.gi * bi, gbi = p.gr * bi + p.gi * br;
    const double gar = p.gr * ar - p.gi * ai, gai = p.gr * ai + p.gi * ar;
    jr = p.c * ar + sj * gbr; ji = p.c * ai + sj * gbi;
    kr = p.c * br + sk * gar; ki = p.c * bi + sk * gai;
}

__global__ void __launch_bounds__(kThreads) kPauliRotVec(double* re, double* im, InsSpec ins,
                                                         uint64_t setMask, uint64_t nThreads, PauliRot p) {
    const uint64_t t = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
    if (t >= nThreads) return;
    const uint64_t j0 = insertZeros(t << 1, ins) | setMask;
    const uint64_t k0 = j0 ^ p.xmask;
    chainStart();
    double2 jr = ld2(re + j0), ji = ld2(im + j0), kr = ld2(re + k0), ki = ld2(im + k0);
    pauliPair(p, j0, jr.x, ji.x, kr.x, ki.x);
    pauliPair(p, j0 + 1, jr.y, ji.y, kr.y, ki.y);
    st2(re + j0, jr); st2(im + j0, ji); st2(re + k0, kr); st2(im + k0, ki);
}

__global__ void __launch_bounds__(kThreads) kPauliRotScalar(double* re, double* im, InsSpec ins,
                                                            uint64_t setMask, uint64_t nPairs, PauliRot p) {
    const uint64_t t = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
    if (t >= nPairs) return;
    const uint64_t j = insertZeros(t, ins) | setMask;
    const uint64_t k = j ^ p.xmask;
    chainStart();
    double jr = re[j], ji = im[j], kr = re[k], ki = im[k];
    pauliPair(p, j, jr, ji, kr, ki);
    re[j] = jr; im[j] = ji; re[k] = kr; im[k] = ki;
}

// ------------------------------------------------------- swap (QuEST_gpu.cu:1737-1769)
__global__ void __launch_bounds__(kThreads) kSwap(double* re, double* im, InsSpec ins,
                                                  uint64_t b1, uint64_t b2, uint64_t n) {
    const uint64_t t = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
    if (t >= n) return;
    const uint64_t base = insertZeros(t, ins);
    const uint64_t a = base | b1, b = base | b2;
    chainStart();
    const double r = re[a], m = im[a];
    re[a] = re[b]; im[a] = im[b];
    re[b] = r; im[b] = m;
}

// ------------------------------------------------------- dense k-qubit matrix
// One block handles G groups of D = 2^k amplitudes; thread (r, g) loads
// amplitude r of group g, then computes row r of M . v_g from shared memory.
// Consecutive threads take consecutive groups so the loads of one row index
// coalesce when the targets are above the low qubits.
__global__ void kMatrixN(double* __restrict__ re, double* __restrict__ im, InsSpec ins, uint64_t setMask,
                         int k, const int* __restrict__ targs, const double* __restrict__ mr,
                         const double* __restrict__ mi, uint64_t nGroups, int G) {
    extern __shared__ double sm[];
    const int D = 1 << k;
    double* vr = sm;
    double* vi = sm + (size_t)D * G;
    const int g = threadIdx.x % G;
    const int r = threadIdx.x / G;
    const uint64_t grp = (uint64_t)blockIdx.x * G + g;
    const bool live = grp < nGroups;
    uint64_t addr = 0;
    if (live) {
        addr = insertZeros(grp, ins) | setMask;
        for (int b = 0; b < k; ++b)
            if (r >> b & 1) addr |= 1ull << targs[b];
        vr[r * G + g] = re[addr];
        vi[r * G + g] = im[addr];
    }
    __syncthreads();
    if (!live) return;
    double sr = 0.0, si = 0.0;
    const double* rowr = mr + (size_t)r * D;
    const double* rowi = mi + (size_t)r * D;
    for (int c = 0; c < D; ++c) {
        const double ar = __ldg(rowr + c), ai = __ldg(rowi + c);
        const double xr = vr[c * G + g], xi = vi[c * G + g];
        sr += ar * xr - ai * xi;
        si += ar * xi + ai * xr;
    }
    re[addr] = sr;
    im[addr] = si;
}

// device staging for gateMatrixN (matrix + targets), grown on demand
double* g_matBuf = nullptr;
size_t g_matCap = 0;

}  // namespace

// --------------------------------------------------------------- launchers
// The plain path of every general 2 x 2 gate.
static void launchMatrix2(SV s, uint64_t ctrl, uint64_t setMask, uint64_t pmask, const Mat2& u, const char* caller) {
    if (g_plainArith == 1) {
        launchPair(s, ctrl, setMask, pmask, matrix2DF(u), caller);
        return;
    }
    // a diagonal matrix (rotateZ, controlledRotateZ) pairs no amplitudes: 120
    // us at 23 qubits as a general one, 45 so
    if (u.r[0][1] == 0 && u.i[0][1] == 0 && u.r[1][0] == 0 && u.i[1][0] == 0) {
        const OpDiag2 d{pmask, u.r[0][0], u.i[0][0], u.r[1][1], u.i[1][1]};
        if (d.dr == d.ar && d.di == -d.ai) launchTurn(s, ctrl, setMask, pmask, d.ar, -d.ai, d, caller);
        else launchDiag(s, ctrl, setMask, d, caller);
        return;
    }
    const OpMatrix2 exact{u};
    // the real form, rows and columns in the order (ur, ui, lr, li)
    double r[4][4];
    for (int i = 0; i < 2; ++i)
        for (int j = 0; j < 2; ++j) {
            r[2 * i][2 * j] = r[2 * i + 1][2 * j + 1] = u.r[i][j];
            r[2 * i][2 * j + 1] = -u.i[i][j];
            r[2 * i + 1][2 * j] = u.i[i][j];
        }
    OpFixed4 f4;
    f4.exact = exact;
    if (fx::mapFits<4>(r, f4.f)) {
        launchPair(s, ctrl, setMask, pmask, f4, caller);
        return;
    }
    // two real 2 x 2 maps: ur with lr (or li), ui with li (or lr)
    for (int cross = 0; cross < 2; ++cross) {
        const int a[2] = {0, cross ? 3 : 2}, b[2] = {1, cross ? 2 : 3};
        bool apart = true;
        for (int i = 0; i < 2; ++i)
            for (int j = 0; j < 2; ++j) apart = apart && r[a[i]][b[j]] == 0 && r[b[i]][a[j]] == 0;
        if (!apart) continue;
        OpFixed2 f2;
        for (int i = 0; i < 2; ++i)
            for (int j = 0; j < 2; ++j) {
                f2.exact.a[i][j] = r[a[i]][a[j]];
                f2.exact.b[i][j] = r[b[i]][b[j]];
            }
        if (fx::mapFits<2>(f2.exact.a, f2.fa) && fx::mapFits<2>(f2.exact.b, f2.fb))
            launchPair(s, ctrl, setMask, pmask, f2, caller, cross);
        else
            launchPair(s, ctrl, setMask, pmask, f2.exact, caller, cross);
        return;
    }
    launchPair(s, ctrl, setMask, pmask, exact, caller);
}

void gateMatrix2(SV s, int target, uint64_t ctrl, uint64_t flip, const Mat2& u) {   // QuEST_gpu.cu:966, 1231, 1299
    if (s.cap) {
        const double ur[4] = {u.r[0][0], u.r[0][1], u.r[1][0], u.r[1][1]}, ui[4] = {u.i[0][0], u.i[0][1], u.i[1][0], u.i[1][1]};
        if (capturePair(s, target, ctrl, flip, ur, ui)) return;
    }
    launchMatrix2(s, ctrl, ctrl & ~flip, 1ull << target, u, "unitary");
}

// QuEST_gpu.cu:783-844: up' = a.up - conj(b).lo ; lo' = b.up + conj(a).lo
void gateCompact(SV s, int target, uint64_t ctrl, double ar, double ai, double br, double bi) {   // QuEST_gpu.cu:838, 905
    if (s.cap) {
        const double ur[4] = {ar, -br, br, ar}, ui[4] = {ai, bi, bi, -ai};     // [alpha, -conj(beta); beta, conj(alpha)]
        if (capturePair(s, target, ctrl, 0, ur, ui)) return;
    }
    const Mat2 m{{{ar, -br}, {br, ar}}, {{ai, bi}, {bi, -ai}}};
    launchMatrix2(s, ctrl, ctrl, 1ull << target, m, "compactUnitary");
}

void gateHadamard(SV s, int target) {                                                // QuEST_gpu.cu:1771-1826
    const double f = 0.70710678118654752440;
    if (s.cap) {
        const double ur[4] = {f, f, f, -f}, ui[4] = {0, 0, 0, 0};
        if (capturePair(s, target, 0, 0, ur, ui)) return;
    }
    const Mat2 m{{{f, f}, {f, -f}}, {{0, 0}, {0, 0}}};
    launchMatrix2(s, 0, 0, 1ull << target, m, "hadamard");
}

bool setPlainArithmetic(int mode) {
    if (mode != 0 && mode != 1) return false;
    g_plainArith = mode;
    return true;
}
int plainArithmetic() { return g_plainArith; }

void gateNot(SV s, uint64_t ctrl, uint64_t targMask) {                               // QuEST_gpu.cu:1354, 1867, 1912
    if (s.cap && captureNot(s, ctrl, targMask)) return;
    launchPair(s, ctrl, ctrl, targMask, OpSwap{}, "controlledNot");
}

void gatePauliY(SV s, int target, uint64_t ctrl, double conjFac) {                   // QuEST_gpu.cu:1387, 1439
    if (s.cap) {
        const double ur[4] = {0, 0, 0, 0}, ui[4] = {0, -conjFac, conjFac, 0};   // [0, -i; i, 0] (conjugated: conjFac = -1)
        if (capturePair(s, target, ctrl, 0, ur, ui)) return;
    }
    launchPair(s, ctrl, ctrl, 1ull << target, OpPauliY{conjFac}, "pauliY");
}

void gatePhase(SV s, uint64_t mask, double tr, double ti) {                          // QuEST_gpu.cu:1485, 1521, 1552, 1702
    if (s.cap && capturePhase(s, mask, tr, ti)) return;
    launchTurn(s, mask, mask, 0, tr, -ti, OpPhase{tr, ti}, "phaseShift");
}

void gateRotateZ(SV s, uint64_t ctrl, uint64_t targ, double angle) {                 // QuEST_gpu.cu:1582, 1615
    if (s.cap && captureRotateZ(s, ctrl, targ, angle)) return;
    const double c = cos(angle / 2), sn = sin(angle / 2);
    launchTurn(s, ctrl, ctrl, targ, c, sn, OpRotZ{targ, c, sn}, "multiRotateZ");
}

void gatePauliRotation(SV s, uint64_t ctrl, uint64_t xmask, uint64_t ymask, uint64_t zmask, double angle, int conj) {
    if (s.cap && capturePauliRotation(s, ctrl, xmask, ymask, zmask, angle, conj)) return;
    if (xmask == 0) {                                      // diagonal: plain Z-rotation on the Y/Z-free mask
        gateRotateZ(s, ctrl, zmask, conj ? -angle : angle);
        return;
    }
    const int nY = __builtin_popcountll(ymask);
    // g = -i * (-i)^nY
    static const double pr[4] = {1, 0, -1, 0}, pi[4] = {0, -1, 0, 1};   // (-i)^m
    const int m = (nY + 1) & 3;
    PauliRot p;
    p.xmask = xmask;
    p.yz = ymask | zmask;
    p.c = cos(angle / 2);
    p.s = sin(angle / 2);
    p.gr = pr[m];
    p.gi = conj ? -pi[m] : pi[m];
    const uint64_t lowBit = xmask & (~xmask + 1ull);
    const uint64_t insMask = ctrl | lowBit;
    const InsSpec ins = makeIns(insMask);
    const int free = s.n - ins.n;
    if (free < 0) return;
    const uint64_t nPairs = 1ull << free;
    cudaStream_t st = stream();
    if (nPairs >= 2 && !(insMask & 1ull) && !(xmask & 1ull))
        chain<kPauliRotVec>(blocksFor(nPairs / 2), kThreads, st, s.re, s.im, ins, ctrl, nPairs / 2, p);
    else
        chain<kPauliRotScalar>(blocksFor(nPairs), kThreads, st, s.re, s.im, ins, ctrl, nPairs, p);
    launchFailed("multiRotatePauli");
}

void gateSwap(SV s, int q1, int q2) {
    if (s.cap && captureSwap(s, q1, q2)) return;
    const InsSpec ins = makeIns((1ull << q1) | (1ull << q2));
    const uint64_t n = 1ull << (s.n - 2);
    chain<kSwap>(blocksFor(n), kThreads, stream(), s.re, s.im, ins, 1ull << q1, 1ull << q2, n);
    launchFailed("swapGate");
}

void gateMatrixN(SV s, uint64_t ctrl, const int* targs, int k, const double* mr, const double* mi) {   // QuEST_gpu.cu:1033, 1166
    if (s.cap && captureMatrixN(s, ctrl, targs, k, mr, mi)) return;
    const int D = 1 << k;
    const size_t matDoubles = 2 * (size_t)D * D;
    const size_t need = matDoubles * sizeof(double) + 64 * sizeof(int);
    if (need > g_matCap) {
        if (g_matBuf) cudaFree(g_matBuf);
        g_matBuf = nullptr;
        g_matCap = 0;
        if (QG_CUDA(cudaMalloc(&g_matBuf, need), "multiQubitUnitary")) return;
        g_matCap = need;
    }
    // pageable sources: cudaMemcpyAsync returns once the host data is staged,
    // so the caller's arrays may be reused immediately.
    std::vector<double> host(matDoubles);
    std::copy(mr, mr + (size_t)D * D, host.begin());
    std::copy(mi, mi + (size_t)D * D, host.begin() + (size_t)D * D);
    int tg[64];
    for (int i = 0; i < k; ++i) tg[i] = targs[i];
    cudaStream_t st = stream();
    if (QG_CUDA(cudaMemcpyAsync(g_matBuf, host.data(), matDoubles * sizeof(double), cudaMemcpyHostToDevice, st), "multiQubitUnitary")) return;
    int* dT = reinterpret_cast<int*>(g_matBuf + matDoubles);
    if (QG_CUDA(cudaMemcpyAsync(dT, tg, k * sizeof(int), cudaMemcpyHostToDevice, st), "multiQubitUnitary")) return;
    uint64_t tmask = 0;
    for (int i = 0; i < k; ++i) tmask |= 1ull << targs[i];
    const InsSpec ins = makeIns(tmask | ctrl);
    const int free = s.n - ins.n;
    if (free < 0) return;
    const uint64_t nGroups = 1ull << free;
    int G = std::max(1, 256 / D);
    if ((uint64_t)G > nGroups) G = (int)nGroups;
    const int threads = G * D;
    const unsigned blocks = (unsigned)((nGroups + G - 1) / G);
    const size_t smem = 2 * (size_t)D * G * sizeof(double);
    if (smem > 48 * 1024) cudaFuncSetAttribute(kMatrixN, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kMatrixN<<<blocks, threads, smem, st>>>(s.re, s.im, ins, ctrl, k, dT, g_matBuf, g_matBuf + (size_t)D * D, nGroups, G);
    launchFailed("multiQubitUnitary");
}

}  // namespace qg

extern "C" {
/* Arithmetic of the plain path's general 2 x 2 gates (compactUnitary and the
 * rotations built on it, unitary and its controlled forms, hadamard): 0 =
 * FP64's precision (the default), 1 = double-float on the FP32 and integer pipes
 * (df64.cuh).  Returns 0, or -1 for an unknown mode. */
int quest_gb300_setPlainArithmetic(int mode) { return qg::setPlainArithmetic(mode) ? 0 : -1; }
int quest_gb300_getPlainArithmetic(void) { return qg::plainArithmetic(); }
}
