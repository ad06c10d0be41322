// pauli_tile.cu -- a sequence of Pauli rotations (a Trotter circuit) on FP64
// amplitudes, many rotations per pass over the state (sm_103a).
//
// One launch per rotation (sv_gates.cu) streams the state once per term and
// spends 16 FP64 operations on a pair of amplitudes: at 22 qubits 67 us a
// term with X or Y and 37 us a diagonal one, bound by the FP64 pipe, against
// 20 us of HBM time.  Here a block keeps a tile of 2^b amplitudes in shared
// memory and applies every rotation of a run whose X/Y qubits are tile qubits
// before it writes the tile back; Z factors are unrestricted, as a sign from
// the tile's fixed qubits.  The FP64 work, which stays the bound, is cut by
//   * merging neighbouring rotations with the same X/Y mask that commute: on
//     a pair they are rotations by +-phi_1 +-phi_2, so X..X and Y..Y of equal
//     weight leave half the pairs alone and turn the others by 2 phi;
//   * three multiply-adds per plane rotation, by lifting: x -= t y; y += s x;
//     x -= t y with t = tan(phi/2), s = sin(phi), where the direct form takes
//     four operations (and rounds once more);
//   * one complex factor per run of diagonal rotations: the terms are dealt
//     to windows of at most 12 qubits, a small kernel tabulates each window's
//     exp(-i sum +-phi) and an amplitude takes the product of its entries.
// Second-order step of an 11-site Fermi-Hubbard chain (22 qubits, 146
// rotations): 8.17 ms one launch a term; here, in 5 passes, 0.61 ms on a state
// without zeros, 0.34 ms from a classical state.
#include "chain_launch.cuh"
#include "qg_internal.h"

#include <algorithm>
#include <cmath>
#include <unordered_map>
#include <vector>

namespace qg {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxTileBits = 12;      // 64 KB of amplitudes: three blocks an SM
constexpr int kLow = 3;               // qubits 0..2 are tile qubits: runs of 64 bytes
constexpr int kMaxOps = 48;
constexpr int kMaxWindows = 4, kWindowBits = 12;
constexpr int kMaxTableTerms = 96;
static_assert(kMaxWindows * (size_t(2) << kWindowBits) <= kPhaseTableDoubles, "phase tables");

enum Kind { kCross, kDirect, kParityPhase, kTablePhase };

// A rotation by angle (-1)^popc(j & m) phi[popc(j & d) & 1] of every pair
// (j, j ^ x) (kCross: its (re j, im k) and (re k, im j); kDirect: (re k, re j)
// and (im k, im j)), or of every amplitude's (im, re) (kParityPhase).  Per
// parity of j & d: t, s, whether the result is negated, whether it does anything.
struct TileOp {
    double t[2], s[2];
    uint64_t m, d;               // the masks' qubits outside the tile
    uint32_t xl, ml, dl;         // tile qubits of x, m, d
    int kind;
    int low;                     // lowest bit of xl
    int fix;                     // only one parity acts: the tile bit of d that is set for it, or -1
    unsigned char neg[2], act[2];
    int w0, w1;                  // kTablePhase: windows
};
struct Window {
    int bits;
    unsigned char pos[kWindowBits];      // its qubits, ascending
    unsigned char local[kWindowBits];    // their tile bits, 255: outside the tile
};
struct TilePass {
    int b, numOps;
    unsigned char pos[kMaxTileBits];     // the tile's qubits, ascending
    double scale;                        // of the amplitudes written back
    TileOp op[kMaxOps];
    Window win[kMaxWindows];
};
struct TableSpec {
    int numWindows;
    int bits[kMaxWindows], first[kMaxWindows + 1];
    uint32_t mask[kMaxTableTerms];       // over the window's bits
    double phi[kMaxTableTerms], lo[kMaxTableTerms];     // phi + lo
    double grow[kMaxWindows];                           // the window's factors are scaled by 1 + grow
};

// Tables (1 + grow) exp(-i sum_k (-1)^popc(index & mask_k) phi_k); the sum is
// compensated (TwoSum), so an entry is as good as one sincos of the exact sum.
__global__ void __launch_bounds__(kThreads) kPhaseTables(const __grid_constant__ TableSpec ts, double2* tab) {
    chainStart();
    const int w = blockIdx.y;
    const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= 1u << ts.bits[w]) return;
    double hi = 0.0, lo = 0.0;
    for (int k = ts.first[w]; k < ts.first[w + 1]; ++k) {
        const double x = (__popc(i & ts.mask[k]) & 1) ? -ts.phi[k] : ts.phi[k];
        const double sum = hi + x, z = sum - hi;
        lo += (hi - (sum - z)) + (x - z);
        lo += (__popc(i & ts.mask[k]) & 1) ? -ts.lo[k] : ts.lo[k];
        hi = sum;
    }
    double s, c;
    sincos(hi, &s, &c);
    const double g = ts.grow[w];
    tab[((size_t)w << kWindowBits) + i] = make_double2(c + (g * c - s * lo), -(s + (g * s + c * lo)));
}

__device__ __forceinline__ double flip(double v, uint32_t sign) {      // sign: 0 or 0x80000000
    return __hiloint2double(__double2hiint(v) ^ (int)sign, __double2loint(v));
}
__device__ __forceinline__ uint32_t bits(double v) {                   // 0 for a zero of either sign
    return ((uint32_t)__double2hiint(v) << 1) | (uint32_t)__double2loint(v);
}
__device__ __forceinline__ void rotate(double& x, double& y, double t, double s, uint32_t neg) {
    const double x1 = fma(-t, y, x), y1 = fma(s, x1, y);
    x = flip(fma(-t, y1, x1), neg);
    y = flip(y1, neg);
}
// The lanes of a warp that take part in a loop of the block's threads over
// `count`, a power of two: all of its warps, or the first lanes of one.
__device__ __forceinline__ uint32_t voters(uint32_t count) { return count >= 32 ? 0xffffffffu : (1u << count) - 1u; }
__device__ __forceinline__ uint32_t insert0(uint32_t k, int b) { return ((k >> b) << (b + 1)) | (k & ((1u << b) - 1u)); }

__global__ void __launch_bounds__(kThreads) kPauliTile(double* re, double* im,
                                                       const __grid_constant__ TilePass p,
                                                       const double2* tables) {
    extern __shared__ double2 sm[];
    const int b = p.b;
    const uint32_t size = 1u << b, sizeVoters = voters(size);
    double* sr = reinterpret_cast<double*>(sm);
    double* si = sr + size;
    uint64_t* high = reinterpret_cast<uint64_t*>(si + size);           // qubits of tile index bits >= kLow
    uint64_t base = blockIdx.x;
    for (int k = 0; k < b; ++k) base = ((base >> p.pos[k]) << (p.pos[k] + 1)) | (base & ((1ull << p.pos[k]) - 1ull));
    for (uint32_t h = threadIdx.x; h < size >> kLow; h += kThreads) {
        uint64_t a = base;
        for (int k = kLow; k < b; ++k) a |= (uint64_t)((h >> (k - kLow)) & 1u) << p.pos[k];
        high[h] = a;
    }
    chainStart();
    __syncthreads();
    for (uint32_t l = 2 * threadIdx.x; l < size; l += 2 * kThreads) {
        const uint64_t a = high[l >> kLow] | (l & ((1u << kLow) - 1u));
        sm[l / 2] = *reinterpret_cast<const double2*>(re + a);
        sm[(size + l) / 2] = *reinterpret_cast<const double2*>(im + a);
    }
    for (int o = 0; o < p.numOps; ++o) {
        __syncthreads();
        const TileOp& op = p.op[o];
        if (op.kind == kTablePhase) {
            for (uint32_t l = threadIdx.x; l < size; l += kThreads) {
                const double x = sr[l], y = si[l];
                if (!__any_sync(sizeVoters, (bits(x) | bits(y)) != 0)) continue;
                double fr = 1.0, fi = 0.0;
                for (int w = op.w0; w < op.w1; ++w) {
                    const Window& win = p.win[w];
                    uint32_t idx = 0;
                    for (int k = 0; k < win.bits; ++k) {
                        const uint32_t bit = win.local[k] != 255 ? l >> win.local[k] : (uint32_t)(base >> win.pos[k]);
                        idx |= (bit & 1u) << k;
                    }
                    const double2 f = tables[((size_t)w << kWindowBits) + idx];
                    if (w == op.w0) {
                        fr = f.x;
                        fi = f.y;
                    } else {
                        const double gr = fr * f.x - fi * f.y;
                        fi = fr * f.y + fi * f.x;
                        fr = gr;
                    }
                }
                sr[l] = fr * x - fi * y;
                si[l] = fr * y + fi * x;
            }
            continue;
        }
        const uint32_t outM = __popcll(base & op.m) & 1, outD = __popcll(base & op.d) & 1;
        if (op.kind == kParityPhase) {
            for (uint32_t l = threadIdx.x; l < size; l += kThreads) {
                const uint32_t sgn = ((__popc(l & op.ml) & 1) ^ outM) << 31;
                double x = sr[l], y = si[l];
                if (!__any_sync(sizeVoters, (bits(x) | bits(y)) != 0)) continue;
                rotate(y, x, flip(op.t[0], sgn), flip(op.s[0], sgn), op.neg[0] ? 0x80000000u : 0u);
                sr[l] = x;
                si[l] = y;
            }
            continue;
        }
        // pairs with bit `low` of the tile index clear; where one parity of
        // j & d alone acts, only its pairs, with bit `fix` set to match
        const int one = op.act[0] && op.act[1] ? -1 : op.act[0] ? 0 : 1;
        if (op.dl == 0 && one >= 0 && (int)outD != one) continue;
        const int fix = op.fix;
        const uint32_t pairs = fix >= 0 ? size / 4 : size / 2, pairVoters = voters(pairs);
        for (uint32_t t = threadIdx.x; t < pairs; t += kThreads) {
            uint32_t j;
            if (fix >= 0) {
                j = insert0(insert0(t, min(op.low, fix)), max(op.low, fix));
                if (((__popc(j & op.dl) & 1) ^ outD) != (uint32_t)one) j |= 1u << fix;
            } else {
                j = insert0(t, op.low);
            }
            const uint32_t k = j ^ op.xl;
            const uint32_t set = (__popc(j & op.dl) & 1) ^ outD;
            const uint32_t sgn = ((__popc(j & op.ml) & 1) ^ outM) << 31;
            const double tt = flip(op.t[set], sgn), ss = flip(op.s[set], sgn);
            const uint32_t neg = op.neg[set] ? 0x80000000u : 0u;
            double jr = sr[j], ji = si[j], kr = sr[k], ki = si[k];
            // zeros stay zeros: a warp whose pairs hold nothing (particle-number
            // sectors leave most of a register zero) spends no FP64 on them
            if (!__any_sync(pairVoters, (bits(jr) | bits(ji) | bits(kr) | bits(ki)) != 0)) continue;
            if (op.kind == kCross) {
                rotate(jr, ki, tt, ss, neg);
                rotate(kr, ji, tt, ss, neg);
            } else {
                rotate(kr, jr, tt, ss, neg);
                rotate(ki, ji, tt, ss, neg);
            }
            sr[j] = jr; si[j] = ji; sr[k] = kr; si[k] = ki;
        }
    }
    __syncthreads();
    for (uint32_t l = 2 * threadIdx.x; l < size; l += 2 * kThreads) {
        const uint64_t a = high[l >> kLow] | (l & ((1u << kLow) - 1u));
        double2 x = sm[l / 2], y = sm[(size + l) / 2];
        if (p.scale != 1.0) {
            x.x *= p.scale; x.y *= p.scale;
            y.x *= p.scale; y.y *= p.scale;
        }
        *reinterpret_cast<double2*>(re + a) = x;
        *reinterpret_cast<double2*>(im + a) = y;
    }
}

// amplitudes, and the qubits of the tile index bits from kLow up
size_t tileShared(int b) { return (size_t(16) << b) + (size_t(8) << (b - kLow)); }

// ------------------------------------------------------------------- planning
struct Sum {                       // an angle as an unevaluated sum of two doubles
    double hi = 0.0, lo = 0.0;
    void add(const Sum& x) {
        const double s = hi + x.hi, z = s - hi;
        lo += (hi - (s - z)) + (x.hi - z) + x.lo;
        hi = s;
    }
    Sum operator-() const { return Sum{-hi, -lo}; }
};

// A rotation is the one of the doubles c = cos(angle / 2), s = sin(angle / 2),
// as every single rotation of the library applies it: a turn by atan2(s, c)
// (angle / 2 + lo) that also scales all amplitudes by hypot(c, s) = 1 + grow.
// A circuit repeats few angles, so that these last bits add up: over the 146
// rotations of a 22-qubit Hubbard step the turns by the exact angles are
// 3e-15 off the product of the rotations, with lo and grow 5e-16.
// An angle of many turns is told by the same c and s as one within half a
// turn, and that one is taken: the sums of merged angles then keep a lo so
// small that its square is nothing.
struct Turn {
    Sum phi;
    double grow;
};
Turn turnOf(double angle) {
    const double a = angle / 2, c = std::cos(a), s = std::sin(a);
    const long double lc = c, ls = s;
    Turn t;
    t.phi.hi = std::fabs(a) > 64 ? std::atan2(s, c) : a;
    long double sh, ch;
    ::sincosl(t.phi.hi, &sh, &ch);
    t.phi.lo = (double)(ls * ch - lc * sh);
    t.grow = (double)((lc * lc + ls * ls - 1) / 2);
    return t;
}

// Neighbouring rotations merged into one step: a pair rotation (x != 0) or a
// run of diagonal ones.
struct Step {
    uint64_t x = 0, m = 0, d = 0;
    bool cross = false, hasD = false;
    Sum even, odd;                                  // angles where popc(j & d) is even, odd
    std::vector<std::pair<uint64_t, Sum>> diag;     // (Z mask, phi)
    double grow = 0;                                // the rotations' scale, less 1
    size_t first = 0, count = 0;                    // the rotations it stands for
};

// phi of a rotation: exp(-i phi P) on a pair is the plane rotation by
// (-1)^popc(j & yz) phi of (re j, im k) for an even number of Y (kCross), of
// (re k, re j) for an odd one
Sum planeAngle(const PauliRotation& r, const Sum& a) {
    const int m = (__builtin_popcountll(r.y) + 1) & 3;     // exp(-i phi P): -i (-i)^nY = (-i)^m
    if (r.x == 0) return r.conj ? -a : a;
    if (m & 1) return (m == 1) != (r.conj != 0) ? -a : a;  // i Im: -1 for m = 1, +1 for m = 3; conjugated
    return m == 0 ? a : -a;
}

void merge(const std::vector<PauliRotation>& seq, std::vector<Step>& steps) {
    std::unordered_map<double, Turn> turns;
    for (size_t i = 0; i < seq.size(); ++i) {
        const PauliRotation& r = seq[i];
        auto at = turns.find(r.angle);
        if (at == turns.end()) at = turns.emplace(r.angle, turnOf(r.angle)).first;
        const Sum phi = planeAngle(r, at->second.phi);
        const double grow = at->second.grow;
        Step* last = steps.empty() ? nullptr : &steps.back();
        if (r.x == 0) {
            if (!last || last->x || last->diag.size() >= kMaxTableTerms) {
                steps.emplace_back();
                last = &steps.back();
                last->first = i;
            }
            auto same = std::find_if(last->diag.begin(), last->diag.end(), [&](auto& t) { return t.first == r.z; });
            if (same != last->diag.end()) same->second.add(phi);
            else last->diag.push_back({r.z, phi});
            last->grow += grow;
            ++last->count;
            continue;
        }
        const uint64_t yz = r.y | r.z;
        const bool cross = !(__builtin_popcountll(r.y) & 1);
        if (last && last->x == r.x && last->cross == cross) {
            // equal X/Y masks commute when the numbers of Y agree in parity
            const uint64_t d = last->m ^ yz;
            if (d == 0 || !last->hasD || d == last->d) {
                if (d && !last->hasD) {
                    last->d = d;
                    last->hasD = true;
                    last->odd = last->even;
                }
                last->even.add(phi);
                if (last->hasD) last->odd.add(d ? -phi : phi);
                last->grow += grow;
                ++last->count;
                continue;
            }
        }
        steps.emplace_back();
        Step& s = steps.back();
        s.x = r.x;
        s.m = yz;
        s.cross = cross;
        s.even.add(phi);
        s.grow = grow;
        s.first = i;
        s.count = 1;
    }
}

// lifting coefficients of a rotation by a; an angle beyond a quarter turn is
// the rotation by half a turn less, negated
void lift(const Sum& a, double& t, double& s, unsigned char& neg, unsigned char& act) {
    double c = std::cos(a.hi) - std::sin(a.hi) * a.lo;
    s = std::sin(a.hi) + std::cos(a.hi) * a.lo;
    neg = c < 0;
    if (neg) {
        c = -c;
        s = -s;
    }
    t = s / (1 + c);
    act = !(s == 0 && t == 0 && !neg);
}

uint32_t localMask(uint64_t mask, const unsigned char* pos, int b) {
    uint32_t l = 0;
    for (int k = 0; k < b; ++k) l |= (uint32_t)(mask >> pos[k] & 1) << k;
    return l;
}

// The windows of a diagonal run (greedy: the window that grows least); a term
// that fits none, or is alone in its own, is a parity phase of its own.
struct Windows {
    std::vector<uint64_t> bits;
    std::vector<std::vector<std::pair<uint64_t, Sum>>> terms;
    std::vector<std::pair<uint64_t, Sum>> alone;
};
Windows windowsOf(const Step& s) {
    Windows w;
    for (const auto& t : s.diag) {
        int best = -1, grow = 99;
        for (size_t k = 0; k < w.bits.size(); ++k) {
            const int all = __builtin_popcountll(w.bits[k] | t.first), g = all - __builtin_popcountll(w.bits[k]);
            if (all <= kWindowBits && g < grow) {
                best = (int)k;
                grow = g;
            }
        }
        if (best < 0 && __builtin_popcountll(t.first) <= kWindowBits && w.bits.size() < kMaxWindows) {
            w.bits.push_back(0);
            w.terms.emplace_back();
            best = (int)w.bits.size() - 1;
        }
        if (best < 0) {
            w.alone.push_back(t);
            continue;
        }
        w.bits[best] |= t.first;
        w.terms[best].push_back(t);
    }
    for (size_t k = 0; k < w.bits.size();) {
        if (w.terms[k].size() > 1) {
            ++k;
            continue;
        }
        w.alone.push_back(w.terms[k][0]);
        w.bits.erase(w.bits.begin() + k);
        w.terms.erase(w.terms.begin() + k);
    }
    return w;
}

struct PassPlan {
    uint64_t tile = 0;                // tile qubits, without the forced low ones
    std::vector<int> steps;
    int ops = 0, windows = 0, terms = 0;
    bool alone = false;               // a step whose X/Y qubits exceed a tile: one launch a rotation
};

std::vector<PassPlan> cut(const std::vector<Step>& steps, const std::vector<Windows>& win, int n, int b) {
    const int low = std::min(kLow, n), room = b - low;
    std::vector<PassPlan> out;
    for (size_t i = 0; i < steps.size(); ++i) {
        const Step& s = steps[i];
        const uint64_t x = s.x >> low << low;
        const int ops = s.x ? 1 : (int)win[i].alone.size() + (win[i].bits.empty() ? 0 : 1);
        const int windows = s.x ? 0 : (int)win[i].bits.size(), terms = s.x ? 0 : (int)s.diag.size();
        if (__builtin_popcountll(x) > room || ops > kMaxOps) {
            out.emplace_back();
            out.back().alone = true;
            out.back().steps.push_back((int)i);
            continue;
        }
        if (out.empty() || out.back().alone || __builtin_popcountll(out.back().tile | x) > room ||
            out.back().ops + ops > kMaxOps || out.back().windows + windows > kMaxWindows ||
            out.back().terms + terms > kMaxTableTerms)
            out.emplace_back();
        PassPlan& p = out.back();
        p.tile |= x;
        p.steps.push_back((int)i);
        p.ops += ops;
        p.windows += windows;
        p.terms += terms;
    }
    return out;
}

double aloneUs(const Step& s, int n) { return s.count * (3 + std::ldexp(1.0, n) * 8 / (numSMs() * 1.65 * 1900)); }
// Expected microseconds: a launch, the state's traffic, and per SM the FP64
// operations of its tiles (1.65 a clock at 1.9 GHz, as measured), a step not
// under its latency.  Small registers take smaller tiles, so that every SM
// has one; large ones the largest, for the fewest passes.
double cost(const std::vector<PassPlan>& plan, const std::vector<Step>& steps, const std::vector<Windows>& win, int n, int b) {
    const double amps = std::ldexp(1.0, n), tiles = std::ldexp(1.0, n - b), sms = numSMs();
    const double rounds = std::ceil(tiles / sms), perAmp = std::ldexp(1.0, b) / (1.65 * 1900);
    double us = 0;
    for (const PassPlan& p : plan) {
        if (p.alone) {
            for (int i : p.steps) us += aloneUs(steps[i], n);
            continue;
        }
        us += 3 + (p.windows ? 3 : 0) + amps * 32 / 5e6;
        for (int i : p.steps) {
            const Step& s = steps[i];
            const bool half = s.hasD && (s.even.hi == 0 || s.odd.hi == 0);       // only one parity turns
            const double ops = s.x ? (half ? 1.5 : 3) : 3.0 * win[i].alone.size() + 4.0 * win[i].bits.size();
            us += std::max(0.35, ops * perAmp) * rounds;
        }
    }
    return us;
}

}  // namespace

void gatePauliSequence(SV s, const std::vector<PauliRotation>& seq, double* tables) {
    const char* caller = "applyTrotterCircuit";
    auto oneByOne = [&]() {
        for (const PauliRotation& r : seq) gatePauliRotation(s, 0, r.x, r.y, r.z, r.angle, r.conj);
    };
    // angles that are not finite: the passes leave zeros as they are, where a
    // rotation by NaN makes them NaN
    if (!std::all_of(seq.begin(), seq.end(), [](const PauliRotation& r) { return std::isfinite(r.angle); })) return oneByOne();
    // one rotation of a small register is not worth a plan (8 qubits 12.3 us, as
    // tiles 14.1; 16 qubits 13.8 and 14.8; 20 qubits 29.3 and 22.3)
    if (seq.size() == 1 && s.n < 18) return oneByOne();
    std::vector<Step> steps;
    merge(seq, steps);
    std::vector<Windows> win(steps.size());
    for (size_t i = 0; i < steps.size(); ++i)
        if (!steps[i].x) win[i] = windowsOf(steps[i]);
    // without tiles, if they come to more
    int b = 0;
    std::vector<PassPlan> plan;
    double best = 0;
    for (const Step& a : steps) best += aloneUs(a, s.n);
    const int low = std::min(kLow, s.n);
    for (int c = std::min(s.n, 7); c <= std::min(s.n, kMaxTileBits); ++c) {
        // (no pass without a step that fits it)
        if (std::none_of(steps.begin(), steps.end(), [&](const Step& a) { return !a.x || __builtin_popcountll(a.x >> low) <= c - low; }))
            continue;
        std::vector<PassPlan> p = cut(steps, win, s.n, c);
        const double us = cost(p, steps, win, s.n, c);
        if (us >= best) continue;
        b = c;
        best = us;
        plan.swap(p);
    }
    // registers of one to three qubits, strings that fit no tile
    if (b < kLow + 1 || std::all_of(plan.begin(), plan.end(), [](const PassPlan& p) { return p.alone; })) return oneByOne();
    cudaStream_t st = stream();
    const size_t smem = tileShared(b);
    if (QG_CUDA(allowShared<kPauliTile>(tileShared(kMaxTileBits)), caller)) return;
    // the scale of all the passes' rotations: with the first phase table, or
    // where there is none as the last pass writes
    double grow = 0;
    const PassPlan* scaled = nullptr;
    for (const PassPlan& pp : plan) {
        if (pp.alone) continue;
        for (int i : pp.steps) grow += steps[i].grow;
        if (!scaled || !scaled->windows) scaled = &pp;
    }
    for (const PassPlan& pp : plan) {
        if (pp.alone) {
            for (int i : pp.steps)
                for (size_t k = steps[i].first; k < steps[i].first + steps[i].count; ++k)
                    gatePauliRotation(s, 0, seq[k].x, seq[k].y, seq[k].z, seq[k].angle, seq[k].conj);
            continue;
        }
        TilePass p{};
        TableSpec ts{};
        p.b = b;
        p.scale = &pp == scaled && !pp.windows ? 1.0 + grow : 1.0;
        if (&pp == scaled) ts.grow[0] = grow;
        uint64_t tile = pp.tile | ((1ull << kLow) - 1);
        for (int q = 0; q < s.n && __builtin_popcountll(tile) < b; ++q) tile |= 1ull << q;
        for (int q = 0, k = 0; q < s.n; ++q)
            if (tile >> q & 1) p.pos[k++] = (unsigned char)q;
        bool any = p.scale != 1.0;
        auto phase = [&](const std::pair<uint64_t, Sum>& t) {
            TileOp& op = p.op[p.numOps++];
            op.kind = kParityPhase;
            op.m = t.first & ~tile;
            op.ml = localMask(t.first, p.pos, b);
            lift(t.second, op.t[0], op.s[0], op.neg[0], op.act[0]);
            any = true;
        };
        for (int i : pp.steps) {
            const Step& stp = steps[i];
            if (!stp.x) {
                if (!win[i].bits.empty()) {
                    TileOp& op = p.op[p.numOps++];
                    op.kind = kTablePhase;
                    op.w0 = ts.numWindows;
                    for (size_t k = 0; k < win[i].bits.size(); ++k) {
                        const int w = ts.numWindows++;
                        Window& wd = p.win[w];
                        for (int q = 0; q < s.n; ++q)
                            if (win[i].bits[k] >> q & 1) {
                                wd.pos[wd.bits] = (unsigned char)q;
                                wd.local[wd.bits++] = tile >> q & 1 ? (unsigned char)__builtin_popcountll(tile & ((1ull << q) - 1)) : 255;
                            }
                        ts.bits[w] = wd.bits;
                        for (const auto& t : win[i].terms[k]) {
                            const int e = ts.first[w + 1] > ts.first[w] ? ts.first[w + 1] : ts.first[w];
                            ts.mask[e] = localMask(t.first, wd.pos, wd.bits);
                            ts.phi[e] = t.second.hi;
                            ts.lo[e] = t.second.lo;
                            ts.first[w + 1] = e + 1;
                        }
                    }
                    op.w1 = ts.numWindows;
                    any = true;
                }
                for (const auto& t : win[i].alone) phase(t);
                continue;
            }
            TileOp op{};
            op.kind = stp.cross ? kCross : kDirect;
            op.m = stp.m & ~tile;
            op.d = stp.d & ~tile;
            op.xl = localMask(stp.x, p.pos, b);
            op.ml = localMask(stp.m, p.pos, b);
            op.dl = localMask(stp.d, p.pos, b);
            op.low = __builtin_ctz(op.xl);
            op.fix = -1;
            lift(stp.even, op.t[0], op.s[0], op.neg[0], op.act[0]);
            if (stp.hasD) lift(stp.odd, op.t[1], op.s[1], op.neg[1], op.act[1]);
            else op.act[1] = 0;
            if (!op.act[0] && !op.act[1]) continue;
            const uint32_t free = op.dl & ~(1u << op.low);
            if (stp.hasD && op.act[0] != op.act[1] && free) op.fix = 31 - __builtin_clz(free);
            p.op[p.numOps++] = op;
            any = true;
        }
        if (!any) continue;
        if (ts.numWindows) {
            int bits = 0;
            for (int w = 0; w < ts.numWindows; ++w) bits = std::max(bits, ts.bits[w]);
            chain<kPhaseTables>(dim3(((1u << bits) + kThreads - 1) / kThreads, ts.numWindows), kThreads, st, ts,
                                reinterpret_cast<double2*>(tables));
            if (launchFailed(caller)) return;
        }
        chainShared<kPauliTile>(1, (unsigned)(1ull << (s.n - b)), kThreads, smem, st, s.re, s.im, p,
                                reinterpret_cast<const double2*>(tables));
        if (launchFailed(caller)) return;
    }
}

}  // namespace qg
