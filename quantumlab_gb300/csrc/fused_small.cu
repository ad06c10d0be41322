// fused_small.cu -- whole plans on small FP32 registers in one launch
// (sm_103a).  No counterpart in the reference.
//
// On a register of 16 qubits the tensor-core applier is all latency: a 6-qubit
// pass has 8 tiles, so 8 CTAs load their operand images and run one tile each,
// 8.9 us a launch (14.9 us from pass to pass with its launch and the
// clearing of its norm record).  Here one cooperative launch
// of a block per SM runs all the passes:
//   * a pass is cut into chunks of 8, 16 or 32 groups of 64 amplitudes, so that
//     all SMs have one; a chunk is a 64 x 64 complex matrix times 64 x GC, in
//     FP32 multiply-adds from shared memory (8 rows x 4 groups a thread, two
//     rows a packed one, the columns dealt to 4 lanes and up to 4 warps);
//   * the next pass's matrix is copied (cp.async) and its addresses are worked
//     out between a block's arrival at the barrier between passes and the
//     last one's; amplitudes stay in L2.
// A pass then takes about its 2 x 0.6 us of loads and barrier plus its
// multiply-adds, 2^n * 256 of them over 152 SMs (0.9 us at 16 qubits), FP32
// with each sum rounded to nearest, where the tensor cores' truncating
// accumulation needs a norm correction.  16 qubits, 19 passes: 283 us before,
// 105 us now (whole pass of the caller); the batch of nine Trotter instances of 16 qubits, 390 passes
// one class after the other before, all classes side by side now: 3.79 ms
// before, 2.26 ms now.
//
// Every wait on the barrier is bounded: a block that gives up sets the error
// flag and ends.
#include "fused_build.h"
#include "fused_small.h"
#include "qg_internal.h"

#include <algorithm>
#include <cstring>
#include <vector>

namespace qg {

bool tcDefaultAppliers();                   // fused_tc.cu

namespace {

constexpr int kD = 64;                       // a pass acts on 6 qubits (narrower ones are widened)
constexpr unsigned long long kBarrierNs = 2000000000ull;

struct Seg {                                 // one pass of one class of registers
    uint64_t state;                          // floats from the base to the class's first register
    uint64_t mat;                            // floats to its first matrix
    uint32_t chunks;                         // over all its registers
    uint32_t each, more;                     // (first of a step) chunks a block, blocks with one more
    int chunkBits;                           // log2 of a register's chunks
    int n;
    unsigned char pos[12];                   // the chunk's qubits, ascending
    unsigned short word[12];                 // what each stands for: a bit of row << 8 | group
};

__device__ __forceinline__ void copy16(void* dst, const void* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copyWait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// wait until `target` blocks have arrived at the barrier; false when that takes too long
__device__ __forceinline__ bool awaitAll(const unsigned* counter, unsigned target) {
    unsigned long long t0 = 0;
    for (int spin = 0;; ++spin) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
        if (v >= target) return true;
        if ((spin & 1023) == 1023) {
            unsigned long long now;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
            if (t0 == 0) t0 = now;
            else if (now - t0 > kBarrierNs) return false;
        }
    }
}

// two floats, the first in the low word
typedef unsigned long long F2;
__device__ __forceinline__ F2 both(float v) {
    F2 r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float half2of(F2 v, int high) { return __uint_as_float((unsigned)(high ? v >> 32 : v)); }

// GC groups a chunk.  Thread = (8 rows, 4 groups, a share of the columns): the
// lanes are 8 row tiles and 4 column shares, the warps GC / 4 group tiles and
// KH further column shares.
constexpr int kThreads = 256;
template <int GC>
struct Shape {
    static constexpr int bits = GC == 32 ? 11 : GC == 16 ? 10 : 9;
    static constexpr int kh = 32 / GC;
    static constexpr int items = GC / 8;     // 16-byte words of a chunk a thread moves
    static constexpr int xs = GC + 4;        // row stride of the staged amplitudes (16-byte aligned)
    static constexpr int ys = GC + 1;        // of the sums: a warp's 8 row tiles x 4 groups in 32 banks
    static constexpr int xPlane = kD * xs, yPlane = kD * ys;
    static constexpr size_t smem = (2 * kD * kD + (2 * xPlane > kh * 2 * yPlane ? 2 * xPlane : kh * 2 * yPlane)) * sizeof(float);
};

template <int GC>
__global__ void __launch_bounds__(kThreads, 1) kSmallPasses(float* __restrict__ re, float* __restrict__ im,
                                                         const float* __restrict__ mats, const Seg* __restrict__ segs,
                                                         int perStep, int step0, int step1,
                                                         unsigned* __restrict__ counters, int* __restrict__ errFlag) {
    using S = Shape<GC>;
    extern __shared__ float4 smem4[];
    float* const g0 = reinterpret_cast<float*>(smem4);           // the matrix: 64 x 64 re, im, column by column
    float* const x0 = g0 + 2 * kD * kD;                          // staged re, im; later the KH column shares' sums
    __shared__ Seg sg[3][kSmallMaxSegs];                         // this step's, the next two's
    __shared__ int alive;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rt = lane & 7, kl = lane >> 3, gt = warp % (GC / 4), kh = warp / (GC / 4);

    const int segWords = (int)sizeof(Seg) / 4 * perStep;         // at most 160
    auto segWord = [&](int step) {
        return tid < segWords && step < step1 ? __ldg(reinterpret_cast<const uint32_t*>(segs + (size_t)step * perStep) + tid) : 0u;
    };
    auto putSegs = [&](int buf, uint32_t w) {
        if (tid < segWords) reinterpret_cast<uint32_t*>(sg[buf])[tid] = w;
    };
    // block b's chunks of a step are [begin(b), begin(b + 1)) of all its segments' chunks
    auto begin = [&](int buf, uint32_t b) { return sg[buf][0].each * b + min(b, sg[buf][0].more); };
    // a chunk: its matrix, and where this thread's words of it lie (word i:
    // plane, amplitudes from the base, row and group of its first amplitude;
    // its others differ by d0, d1, both)
    struct Chunk {
        uint64_t mat, at[S::items];
        uint32_t word[S::items], d0, d1;     // row << 8 | group
    };
    auto offset = [](uint32_t word, int stride) { return (word >> 8) * stride + (word & 255u); };
    auto chunk = [&](int buf, uint32_t c) {
        int s = 0;
        while (c >= sg[buf][s].chunks) c -= sg[buf][s++].chunks;
        const Seg& g = sg[buf][s];
        const uint32_t inst = c >> g.chunkBits;
        uint32_t base = c & ((1u << g.chunkBits) - 1u);
        Chunk k;
        k.mat = g.mat + (uint64_t)inst * (2 * kD * kD);
        for (int i = 0; i < S::bits; ++i) base = ((base >> g.pos[i]) << (g.pos[i] + 1)) | (base & ((1u << g.pos[i]) - 1u));
        k.d0 = g.word[0];
        k.d1 = g.word[1];
#pragma unroll
        for (int w = 0; w < S::items; ++w) {
            const uint32_t q = 4 * ((uint32_t)(tid + w * kThreads) % (1u << (S::bits - 2)));
            uint32_t off = 0, word = 0;
            for (int i = 2; i < S::bits; ++i) {
                const uint32_t bit = (q >> i) & 1u;
                off |= bit << g.pos[i];
                word += bit * g.word[i];
            }
            k.at[w] = g.state + ((uint64_t)inst << g.n) + (base | off);
            k.word[w] = word;
        }
        return k;
    };
    auto planeOf = [&](int w) { return (int)((tid + w * kThreads) >> (S::bits - 2)); };      // 0 re, 1 im
    auto fetchMatrix = [&](uint64_t at) {
        const float4* src = reinterpret_cast<const float4*>(mats + at);
        float4* dst = reinterpret_cast<float4*>(g0);
#pragma unroll
        for (int i = 0; i < 2 * kD * kD / 4 / kThreads; ++i) copy16(dst + tid + i * kThreads, src + tid + i * kThreads);
    };

    if (tid == 0) alive = 1;
    putSegs(0, segWord(step0));
    putSegs(1, segWord(step0 + 1));
    __syncthreads();
    uint32_t c0, c1;
    Chunk cur{};
    unsigned long long loaded = ~0ull;                           // the matrix in the buffer
    int sb = 0;
    c0 = begin(0, blockIdx.x);
    c1 = begin(0, blockIdx.x + 1);
    if (c0 < c1) {
        cur = chunk(0, c0);
        loaded = cur.mat;
        fetchMatrix(loaded);
    }
    for (int step = step0; step < step1; ++step) {
        const int sn = sb == 2 ? 0 : sb + 1, sa = sn == 2 ? 0 : sn + 1;
        const uint32_t ahead = segWord(step + 2);                // stored once the chunks are done
        float4 v[S::items];
        auto load = [&](const Chunk& k) {
#pragma unroll
            for (int w = 0; w < S::items; ++w)
                v[w] = __ldcg(reinterpret_cast<const float4*>((planeOf(w) ? im : re) + k.at[w]));
        };
        if (c0 < c1) load(cur);
        for (uint32_t c = c0; c < c1; ++c) {
            if (cur.mat != loaded) {
                loaded = cur.mat;
                fetchMatrix(loaded);
            }
#pragma unroll
            for (int w = 0; w < S::items; ++w) {
                float* x = x0 + planeOf(w) * S::xPlane + offset(cur.word[w], S::xs);
                const uint32_t d0 = offset(cur.d0, S::xs), d1 = offset(cur.d1, S::xs);
                x[0] = v[w].x; x[d0] = v[w].y; x[d1] = v[w].z; x[d0 + d1] = v[w].w;
            }
            copyWait();
            __syncthreads();
            Chunk after = cur;                                   // the next chunk's amplitudes come behind the sums
            if (c + 1 < c1) {
                after = chunk(sb, c + 1);
                load(after);
            }
            const float* gr = g0 + 4 * rt;
            const float* px = x0 + 4 * gt;
            // two rows a packed multiply-add: pair r is rows 4 rt + 2 r, + 1
            // (r < 2), 32 + 4 rt + 2 (r - 2), + 1; by group
            F2 ar[4][4] = {}, ai[4][4] = {};
#pragma unroll 2
            for (int jj = 0; jj < kD / (4 * S::kh); ++jj) {
                const int j = (jj * S::kh + kh) * 4 + kl;
                const float* g = gr + j * kD;
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(g), b = *reinterpret_cast<const ulonglong2*>(g + 32);
                const ulonglong2 d = *reinterpret_cast<const ulonglong2*>(g + kD * kD), e = *reinterpret_cast<const ulonglong2*>(g + kD * kD + 32);
                const float4 x4 = *reinterpret_cast<const float4*>(px + j * S::xs), y4 = *reinterpret_cast<const float4*>(px + S::xPlane + j * S::xs);
                const F2 m[4] = {a.x, a.y, b.x, b.y}, n[4] = {d.x, d.y, e.x, e.y};
                const F2 x[4] = {both(x4.x), both(x4.y), both(x4.z), both(x4.w)};
                const F2 y[4] = {both(y4.x), both(y4.y), both(y4.z), both(y4.w)};
                const F2 z[4] = {both(-y4.x), both(-y4.y), both(-y4.z), both(-y4.w)};
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        ar[r][u] = fma2(m[r], x[u], ar[r][u]);
                        ai[r][u] = fma2(m[r], y[u], ai[r][u]);
                        ar[r][u] = fma2(n[r], z[u], ar[r][u]);
                        ai[r][u] = fma2(n[r], x[u], ai[r][u]);
                    }
            }
            // sum over the lanes' column shares: a lane ends with one group
            // (halves by lane bit 4, then by bit 3) of its 8 rows
            const int hi = kl >> 1, lo = kl & 1;
            float sr[8], si[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                float qr[4], qi[4], kr[2], ki[2];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    qr[u] = half2of(ar[r / 2][u], r & 1);
                    qi[u] = half2of(ai[r / 2][u], r & 1);
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    kr[u] = (hi ? qr[u + 2] : qr[u]) + __shfl_xor_sync(0xffffffffu, hi ? qr[u] : qr[u + 2], 16);
                    ki[u] = (hi ? qi[u + 2] : qi[u]) + __shfl_xor_sync(0xffffffffu, hi ? qi[u] : qi[u + 2], 16);
                }
                sr[r] = (lo ? kr[1] : kr[0]) + __shfl_xor_sync(0xffffffffu, lo ? kr[0] : kr[1], 8);
                si[r] = (lo ? ki[1] : ki[0]) + __shfl_xor_sync(0xffffffffu, lo ? ki[0] : ki[1], 8);
            }
            __syncthreads();
            float* out = x0 + kh * 2 * S::yPlane + 4 * gt + kl;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const int row = (r < 4 ? 4 * rt + r : 32 + 4 * rt + r - 4) * S::ys;
                out[row] = sr[r];
                out[S::yPlane + row] = si[r];
            }
            __syncthreads();
#pragma unroll
            for (int w = 0; w < S::items; ++w) {
                const float* x = x0 + planeOf(w) * S::yPlane + offset(cur.word[w], S::ys);
                const uint32_t d0 = offset(cur.d0, S::ys), d1 = offset(cur.d1, S::ys);
                float4 t = make_float4(x[0], x[d0], x[d1], x[d0 + d1]);
#pragma unroll
                for (int k = 1; k < S::kh; ++k) {
                    x += 2 * S::yPlane;
                    t.x += x[0]; t.y += x[d0]; t.z += x[d1]; t.w += x[d0 + d1];
                }
                *reinterpret_cast<float4*>((planeOf(w) ? im : re) + cur.at[w]) = t;
            }
            __syncthreads();
            cur = after;
        }
        if (step + 1 == step1) break;
        // while the other blocks arrive: the next step's first chunk, the copy
        // of its matrix
        if (tid == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counters) : "memory");
        putSegs(sa, ahead);
        sb = sn;
        c0 = begin(sb, blockIdx.x);
        c1 = begin(sb, blockIdx.x + 1);
        if (c0 < c1) {
            cur = chunk(sb, c0);
            if (cur.mat != loaded) {
                loaded = cur.mat;
                fetchMatrix(loaded);
            }
        }
        if (tid == 0 && !awaitAll(counters, (unsigned)(step - step0 + 1) * gridDim.x)) {
            alive = 0;
            *errFlag = 7;
        }
        __syncthreads();
        if (!alive) break;
    }
    copyWait();
    // the last block to end clears both counters for the next launch
    if (tid == 0 && alive) {
        unsigned* ended = counters + 1;
        __threadfence();
        if (atomicAdd(ended, 1u) == gridDim.x - 1) {
            *counters = 0u;
            *ended = 0u;
        }
    }
}

}  // namespace

int smallGroups(uint64_t amps) {
    const uint64_t groups = amps / kD, sms = (uint64_t)numSMs();
    return groups / 16 <= sms / 2 ? 8 : groups / 32 <= sms / 2 ? 16 : 32;
}

bool smallFits(int n, const std::vector<int>& targets) {
    return n >= 10 && n <= 30 && !targets.empty() && targets.size() <= 6;
}

// a pass's qubits, filled up to six with the lowest others
static std::vector<int> widened(std::vector<int> t, int n) {
    for (int q = 0; q < n && (int)t.size() < 6; ++q)
        if (std::find(t.begin(), t.end(), q) == t.end()) t.push_back(q);
    std::sort(t.begin(), t.end());
    return t;
}

size_t smallAddPass(SmallProgram& p, const FusedPass& pass, int n, size_t stateOffset, int registers, size_t mat) {
    const std::vector<int> t = widened(pass.targets, n);
    std::vector<int> all = t;
    const int bits = p.groups == 32 ? 11 : p.groups == 16 ? 10 : 9;
    for (int q = 0; (int)all.size() < bits; ++q)
        if (std::find(t.begin(), t.end(), q) == t.end()) all.push_back(q);
    std::sort(all.begin(), all.end());
    SmallSeg s{};
    s.state = stateOffset;
    s.mat = mat;
    s.chunkBits = n - bits;
    s.chunks = (uint32_t)registers << s.chunkBits;
    s.n = n;
    int row = 0, group = 0;
    for (int i = 0; i < bits; ++i) {
        s.pos[i] = (unsigned char)all[i];
        const bool target = std::find(t.begin(), t.end(), all[i]) != t.end();
        s.word[i] = (unsigned short)(target ? 256 << row++ : 1 << group++);
    }
    p.segs.push_back(s);
    return mat + (size_t)registers * 2 * kD * kD;
}

void smallMatrix(const FusedPass& pass, int n, float* out) {
    const std::vector<int> t = widened(pass.targets, n);
    const int Dk = 1 << pass.targets.size();
    int old[kD], rest[kD];                    // a 6-qubit index's bits on the pass's own qubits, and the others
    for (int i = 0; i < kD; ++i) {
        old[i] = rest[i] = 0;
        for (int b = 0, ob = 0; b < 6; ++b) {
            const bool own = std::find(pass.targets.begin(), pass.targets.end(), t[b]) != pass.targets.end();
            if (own) old[i] |= (i >> b & 1) << ob++;
            else rest[i] |= (i >> b & 1) << b;
        }
    }
    for (int j = 0; j < kD; ++j)
        for (int r = 0; r < kD; ++r) {
            const cplx v = rest[r] == rest[j] ? pass.m[(size_t)old[r] * Dk + old[j]] : cplx(0, 0);
            out[j * kD + r] = (float)v.real();
            out[kD * kD + j * kD + r] = (float)v.imag();
        }
}

bool smallLaunch(const SmallProgram& p, float* re, float* im, int step0, int step1, int* errFlag, cudaStream_t st, const char* caller) {
    static_assert(sizeof(Seg) == sizeof(SmallSeg), "device layout");
    if (step0 >= step1) return true;
    const Seg* segs = reinterpret_cast<const Seg*>(p.dSegs);
    const float* mats = p.dMats;
    int perStep = p.perStep;
    unsigned* counters = p.counters;
    void* args[] = {&re, &im, &mats, &segs, &perStep, &step0, &step1, &counters, &errFlag};
    const void* fn = p.groups == 32 ? (const void*)kSmallPasses<32> : p.groups == 16 ? (const void*)kSmallPasses<16>
                                                                                  : (const void*)kSmallPasses<8>;
    const size_t smem = p.groups == 32 ? Shape<32>::smem : p.groups == 16 ? Shape<16>::smem : Shape<8>::smem;
    if (QG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), caller)) return false;
    if (QG_CUDA(cudaLaunchCooperativeKernel(fn, dim3(p.grid), dim3(kThreads), args, smem, st), caller)) return false;
    return !launchFailed(caller);
}

bool smallUpload(SmallProgram& p, const float* mats, size_t matFloats, const char* caller) {
    // every step's segments at the same stride (absent ones have no chunks)
    const size_t steps = p.first.size() - 1;
    p.perStep = 1;
    for (size_t s = 0; s < steps; ++s) p.perStep = std::max(p.perStep, p.first[s + 1] - p.first[s]);
    if (p.perStep > kSmallMaxSegs) return false;
    std::vector<SmallSeg> segs(steps * p.perStep);
    memset(segs.data(), 0, segs.size() * sizeof(SmallSeg));
    p.maxChunks = 0;
    for (size_t s = 0; s < steps; ++s) {
        uint32_t c = 0;
        for (int i = p.first[s]; i < p.first[s + 1]; ++i) {
            segs[s * p.perStep + (i - p.first[s])] = p.segs[i];
            c += p.segs[i].chunks;
        }
        p.maxChunks = std::max(p.maxChunks, c);
        segs[s * p.perStep].each = c;                // (its total, for now)
    }
    p.grid = std::max(1u, std::min((unsigned)numSMs(), p.maxChunks));
    for (size_t s = 0; s < steps; ++s) {
        SmallSeg& g = segs[s * p.perStep];
        g.more = g.each % p.grid;
        g.each /= p.grid;
    }
    const size_t segBytes = segs.size() * sizeof(SmallSeg), segAt = matFloats * sizeof(float);
    const size_t countersAt = segAt + (segBytes + 31) / 32 * 32, counterBytes = 2 * sizeof(unsigned);
    if (p.bytes < countersAt + counterBytes) {
        smallFree(p);
        if (QG_CUDA(cudaMalloc(&p.buffer, countersAt + counterBytes), caller)) return false;
        p.bytes = countersAt + counterBytes;
    }
    char* b = reinterpret_cast<char*>(p.buffer);
    p.dMats = reinterpret_cast<float*>(b);
    p.dSegs = b + segAt;
    p.counters = reinterpret_cast<unsigned*>(b + countersAt);
    // pageable sources: a copy returns once its source is staged
    return (!mats || !QG_CUDA(cudaMemcpyAsync(p.dMats, mats, segAt, cudaMemcpyHostToDevice, stream()), caller)) &&
           !QG_CUDA(cudaMemcpyAsync(p.dSegs, segs.data(), segBytes, cudaMemcpyHostToDevice, stream()), caller) &&
           !QG_CUDA(cudaMemsetAsync(p.counters, 0, counterBytes, stream()), caller);
}

// after an error: a launch that gave up leaves the counters as they stood
void smallReset(SmallProgram& p) { cudaMemsetAsync(p.counters, 0, 2 * sizeof(unsigned), stream()); }

void smallFree(SmallProgram& p) {
    if (p.buffer) cudaFree(p.buffer);
    p.buffer = nullptr;
    p.bytes = 0;
}

// ------------------------------------------------------------ a plan on one register
namespace {
struct PlanProgram {
    SmallProgram p;
    BuildScratch scratch;                     // of products formed on the device
    int* errFlag = nullptr;                   // page-locked: a kernel writes it only when it gives up
};
}  // namespace

bool smallPlanFits(const FusedPlan& plan) {
    if (plan.numQubits > kSmallMaxQubits || plan.passes.empty() || !tcDefaultAppliers()) return false;
    for (const FusedPass& pass : plan.passes)
        if (!pass.controls.empty() || !smallFits(plan.numQubits, pass.targets)) return false;
    return true;
}

void* smallPlanUpload(const FusedPlan& plan, void* reuse) {
    PlanProgram* pp = reinterpret_cast<PlanProgram*>(reuse);
    if (!pp) pp = new PlanProgram();
    const int n = plan.numQubits;
    pp->p.segs.clear();
    pp->p.first.clear();
    pp->p.groups = smallGroups((uint64_t)1 << n);
    size_t at = 0;
    pp->p.first.push_back(0);
    for (const FusedPass& pass : plan.passes) {
        at = smallAddPass(pp->p, pass, n, 0, 1, at);
        pp->p.first.push_back((int)pp->p.segs.size());
    }
    std::vector<float> mats;
    std::vector<int> deferred;
    std::vector<BuildOutput> outputs;
    for (size_t i = 0; i < plan.passes.size(); ++i) {
        const FusedPass& pass = plan.passes[i];
        if (pass.m.empty()) {
            BuildOutput o;
            o.small = i * 2 * kD * kD;
            const std::vector<int> t = widened(pass.targets, n);
            for (int b = 0; b < 6; ++b)
                if (std::binary_search(pass.targets.begin(), pass.targets.end(), t[b])) o.smallMask |= 1 << b;
            deferred.push_back((int)i);
            outputs.push_back(o);
            continue;
        }
        mats.resize(at);
        smallMatrix(pass, n, mats.data() + i * 2 * kD * kD);
    }
    const char* caller = "applyPlanF32";
    if ((!pp->errFlag && QG_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&pp->errFlag), sizeof(int), cudaHostAllocMapped), caller)) ||
        !smallUpload(pp->p, mats.empty() ? nullptr : mats.data(), at, caller) ||
        !queueBuild(plan, deferred, outputs, pp->p.dMats, pp->scratch, stream(), caller)) {
        smallPlanFree(pp);
        return nullptr;
    }
    *pp->errFlag = 0;
    return pp;
}

void smallPlanFree(void* h) {
    PlanProgram* pp = reinterpret_cast<PlanProgram*>(h);
    if (!pp) return;
    cudaStreamSynchronize(stream());
    smallFree(pp->p);
    freeBuildScratch(pp->scratch);
    if (pp->errFlag) cudaFreeHost(pp->errFlag);
    delete pp;
}

// passes [first, last) of the plan; 0, a kernel's error code, or -1 when the launch failed
int smallPlanApply(void* h, float* re, float* im, int first, int last) {
    PlanProgram* pp = reinterpret_cast<PlanProgram*>(h);
    if (!smallLaunch(pp->p, re, im, first, last, pp->errFlag, stream(), "applyPlanF32")) return -1;
    if (QG_CUDA(cudaStreamSynchronize(stream()), "applyPlanF32")) return -1;
    const int e = *reinterpret_cast<volatile int*>(pp->errFlag);
    if (e) {
        *pp->errFlag = 0;
        smallReset(pp->p);
    }
    return e;
}

}  // namespace qg
