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
// At 16 qubits a pass is some 6000 clocks: loads 600, the 64 x 8 sums 1500
// (1024 at the FP32 rate), their shuffles and stores 1000, the fence and
// barrier 2900.  Sums are FP32 rounded to nearest, where the tensor cores
// truncate and need a norm correction.  19 passes, the caller's whole step with
// its copies: 285 -> 100 us.
//
// Every wait on the barrier is bounded: a block that gives up sets the error
// flag and ends.
#include "chain_launch.cuh"
#include "fused_build.h"
#include "fused_small.h"
#include "qg_internal.h"

#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

namespace qg {

bool tcDefaultAppliers();                   // fused_tc.cu

namespace {

constexpr int kD = 64;                       // a pass acts on 6 qubits (narrower ones are widened)
constexpr unsigned long long kBarrierNs = 2000000000ull;

struct Seg {                                 // a pass
    uint64_t mat;                            // floats to its matrix
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
                                                         uint32_t chunks, int step0, int step1,
                                                         unsigned* __restrict__ counters, int* __restrict__ errFlag) {
    using S = Shape<GC>;
    extern __shared__ float4 smem4[];
    float* const g0 = reinterpret_cast<float*>(smem4);           // the matrix: 64 x 64 re, im, column by column
    float* const x0 = g0 + 2 * kD * kD;                          // staged re, im; later the KH column shares' sums
    __shared__ Seg sg[3];                                        // this step's, the next two's
    __shared__ int alive;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rt = lane & 7, kl = lane >> 3, gt = warp % (GC / 4), kh = warp / (GC / 4);

    constexpr int segWords = (int)sizeof(Seg) / 4;
    auto segWord = [&](int step) {
        return tid < segWords && step < step1 ? __ldg(reinterpret_cast<const uint32_t*>(segs + step) + tid) : 0u;
    };
    auto putSegs = [&](int buf, uint32_t w) {
        if (tid < segWords) reinterpret_cast<uint32_t*>(sg + buf)[tid] = w;
    };
    // this block's chunks of a pass
    const uint32_t each = chunks / gridDim.x, more = chunks % gridDim.x;
    const uint32_t c0 = each * blockIdx.x + min(blockIdx.x, more), c1 = c0 + each + (blockIdx.x < more ? 1 : 0);
    // a chunk: its matrix, and where this thread's words of it lie (word i:
    // plane, amplitudes from the base, row and group of its first amplitude;
    // its others differ by d0, d1, both)
    struct Chunk {
        uint64_t mat, at[S::items];
        uint32_t word[S::items], d0, d1;     // row << 8 | group
    };
    auto offset = [](uint32_t word, int stride) { return (word >> 8) * stride + (word & 255u); };
    auto chunk = [&](int buf, uint32_t c) {
        const Seg& g = sg[buf];
        uint32_t base = c;
        Chunk k;
        k.mat = g.mat;
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
            k.at[w] = base | off;
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
    // (every block has a chunk: the grid is no larger)
    Chunk cur = chunk(0, c0);
    int sb = 0;
    fetchMatrix(cur.mat);
    for (int step = step0; step < step1; ++step) {
        const int sn = sb == 2 ? 0 : sb + 1, sa = sn == 2 ? 0 : sn + 1;
        const uint32_t ahead = segWord(step + 2);                // stored once the chunks are done
        float4 v[S::items];
        auto load = [&](const Chunk& k) {
#pragma unroll
            for (int w = 0; w < S::items; ++w)
                v[w] = __ldcg(reinterpret_cast<const float4*>((planeOf(w) ? im : re) + k.at[w]));
        };
        load(cur);
        for (uint32_t c = c0; c < c1; ++c) {
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
        cur = chunk(sb, c0);
        fetchMatrix(cur.mat);
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

// a pass's qubits, filled up to six with the lowest others
static std::vector<int> widened(std::vector<int> t, int n) {
    for (int q = 0; q < n && (int)t.size() < 6; ++q)
        if (std::find(t.begin(), t.end(), q) == t.end()) t.push_back(q);
    std::sort(t.begin(), t.end());
    return t;
}

static Seg segOf(const FusedPass& pass, int n, int groups, size_t mat) {
    const std::vector<int> t = widened(pass.targets, n);
    std::vector<int> all = t;
    const int bits = groups == 32 ? 11 : groups == 16 ? 10 : 9;
    for (int q = 0; (int)all.size() < bits; ++q)
        if (std::find(t.begin(), t.end(), q) == t.end()) all.push_back(q);
    std::sort(all.begin(), all.end());
    Seg s{};
    s.mat = mat;
    int row = 0, group = 0;
    for (int i = 0; i < bits; ++i) {
        s.pos[i] = (unsigned char)all[i];
        const bool target = std::find(t.begin(), t.end(), all[i]) != t.end();
        s.word[i] = (unsigned short)(target ? 256 << row++ : 1 << group++);
    }
    return s;
}

// the pass's matrix as the kernel reads it, into zeros
static void smallMatrix(const FusedPass& pass, int n, float* out) {
    const std::vector<int> t = widened(pass.targets, n);
    const int Dk = 1 << pass.targets.size();
    // 6-qubit indices by their bits on the other qubits and on the pass's own
    int at[kD];
    for (int i = 0; i < kD; ++i) {
        int own = 0, rest = 0;
        for (int b = 0, ob = 0, rb = 0; b < 6; ++b) {
            if (std::binary_search(pass.targets.begin(), pass.targets.end(), t[b])) own |= (i >> b & 1) << ob++;
            else rest |= (i >> b & 1) << rb++;
        }
        at[rest * Dk + own] = i;
    }
    for (int e = 0; e < kD; e += Dk)
        for (int r = 0; r < Dk; ++r)
            for (int j = 0; j < Dk; ++j) {
                const cplx v = pass.m[(size_t)r * Dk + j];
                float* o = out + at[e + j] * kD + at[e + r];
                o[0] = (float)v.real();
                o[kD * kD] = (float)v.imag();
            }
}

// ------------------------------------------------------------ a plan on one register
namespace {
struct PlanProgram {
    int groups = 16;                          // groups of 64 amplitudes a chunk
    uint32_t chunks = 0;
    BuildScratch scratch;                     // of products formed on the device
    UploadSource source;                      // of the buffer's contents
    int* errFlag = nullptr;                   // page-locked: a kernel writes it only when it gives up
    size_t bytes = 0;                         // room in buffer
    char* buffer = nullptr;                   // device: matrices, passes, barrier counters
    float* mats = nullptr;
    Seg* segs = nullptr;
    unsigned* counters = nullptr;             // arrivals at the barrier, ended blocks; zero between launches
};
constexpr size_t kCounterBytes = 2 * sizeof(unsigned);

template <int GC>
bool launchPasses(void** args, unsigned grid, cudaStream_t st, const char* caller) {
    constexpr size_t smem = Shape<GC>::smem;
    return !QG_CUDA(allowShared<kSmallPasses<GC>>(smem), caller) &&
           !QG_CUDA(cudaLaunchCooperativeKernel((const void*)kSmallPasses<GC>, dim3(grid), dim3(kThreads), args, smem, st), caller);
}
bool launch(const PlanProgram& p, float* re, float* im, int step0, int step1, cudaStream_t st, const char* caller) {
    if (step0 >= step1) return true;
    const Seg* segs = p.segs;
    const float* mats = p.mats;
    uint32_t chunks = p.chunks;
    unsigned* counters = p.counters;
    int* errFlag = p.errFlag;
    void* args[] = {&re, &im, &mats, &segs, &chunks, &step0, &step1, &counters, &errFlag};
    const unsigned grid = std::min((unsigned)numSMs(), chunks);
    const bool ok = p.groups == 32   ? launchPasses<32>(args, grid, st, caller)
                    : p.groups == 16 ? launchPasses<16>(args, grid, st, caller)
                                     : launchPasses<8>(args, grid, st, caller);
    return ok && !launchFailed(caller);
}

// the most of 8, 16, 32 groups a chunk that leaves at most half the SMs
// without a chunk
int groupsFor(uint64_t amps) {
    const uint64_t groups = amps / kD, sms = (uint64_t)numSMs();
    return groups / 16 <= sms / 2 ? 8 : groups / 32 <= sms / 2 ? 16 : 32;
}
}  // namespace

// Page-locked error words, given out by the page: a page-locked allocation and
// its release for each plan took 150 us of a small plan's first application
// (10 qubits, one layer: 296 us with the plan on passes of their own).  The
// first page is kept for the process; when it is full, plans allocate a word of
// their own.
namespace {
class ErrorWords {
public:
    int* take(const char* caller) {
        std::lock_guard<std::mutex> lk(mutex_);
        if (!page_) {
            if (QG_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&page_), kWords * sizeof(int), cudaHostAllocMapped), caller)) {
                page_ = nullptr;
                return nullptr;
            }
            for (int i = kWords; i-- > 0;) free_.push_back(i);
        }
        int* word = nullptr;
        if (!free_.empty()) {
            word = page_ + free_.back();
            free_.pop_back();
        } else if (QG_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&word), sizeof(int), cudaHostAllocMapped), caller)) {
            return nullptr;
        }
        *word = 0;
        return word;
    }
    void give(int* word) {
        std::lock_guard<std::mutex> lk(mutex_);
        if (page_ && word >= page_ && word < page_ + kWords) free_.push_back((int)(word - page_));
        else cudaFreeHost(word);
    }

private:
    static constexpr int kWords = 1024;
    std::mutex mutex_;
    int* page_ = nullptr;
    std::vector<int> free_;
};
ErrorWords& errorWords() {
    static ErrorWords* words = new ErrorWords();     // (outlives every plan)
    return *words;
}
}  // namespace

bool smallPlanFits(const FusedPlan& plan) {
    // a flush of one pass is not worth an upload (19 qubits 82 us, so 91)
    if (plan.deferProducts && plan.passes.size() == 1) return false;
    if (plan.numQubits < 10 || plan.numQubits > kSmallMaxQubits || plan.passes.empty() || !tcDefaultAppliers()) return false;
    for (const FusedPass& pass : plan.passes)
        if (!pass.controls.empty() || pass.targets.empty() || pass.targets.size() > 6) return false;
    return true;
}

void* smallPlanUpload(const FusedPlan& plan, void* reuse) {
    PlanProgram* pp = reinterpret_cast<PlanProgram*>(reuse);
    if (!pp) pp = new PlanProgram();
    const int n = plan.numQubits;
    pp->groups = groupsFor((uint64_t)1 << n);
    pp->chunks = (uint32_t)(((uint64_t)1 << n) / kD / pp->groups);
    const size_t at = plan.passes.size() * 2 * kD * kD;
    std::vector<Seg> segs;
    for (size_t i = 0; i < plan.passes.size(); ++i) segs.push_back(segOf(plan.passes[i], n, pp->groups, i * 2 * kD * kD));
    const char* caller = "applyPlanF32";
    const size_t matBytes = at * sizeof(float), segBytes = (segs.size() * sizeof(Seg) + 31) / 32 * 32;
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
        }
    }
    // the buffer's contents: matrices (none, when the device forms them all),
    // passes, counters at zero
    const size_t matHost = deferred.size() < plan.passes.size() ? matBytes : 0;
    char* host = pp->source.open(matHost + segBytes + kCounterBytes, caller);
    if (!host) {
        smallPlanFree(pp);
        return nullptr;
    }
    for (size_t i = 0; i < plan.passes.size(); ++i)
        if (!plan.passes[i].m.empty()) smallMatrix(plan.passes[i], n, reinterpret_cast<float*>(host) + i * 2 * kD * kD);
    memcpy(host + matHost, segs.data(), segs.size() * sizeof(Seg));
    if (!pp->errFlag && !(pp->errFlag = errorWords().take(caller))) {
        smallPlanFree(pp);
        return nullptr;
    }
    if (pp->bytes < matBytes + segBytes + kCounterBytes) {
        if (pp->buffer) cudaFree(pp->buffer);
        pp->buffer = nullptr;
        pp->bytes = 0;
        if (QG_CUDA(cudaMalloc(&pp->buffer, matBytes + segBytes + kCounterBytes), caller)) {
            smallPlanFree(pp);
            return nullptr;
        }
        pp->bytes = matBytes + segBytes + kCounterBytes;
    }
    pp->mats = reinterpret_cast<float*>(pp->buffer);
    pp->segs = reinterpret_cast<Seg*>(pp->buffer + matBytes);
    pp->counters = reinterpret_cast<unsigned*>(pp->buffer + matBytes + segBytes);
    if (!pp->source.copy(pp->buffer + (matBytes - matHost), stream(), caller) ||
        !queueBuild(plan, deferred, outputs, pp->mats, pp->scratch, stream(), caller)) {
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
    pp->source.release();
    if (pp->buffer) cudaFree(pp->buffer);
    freeBuildScratch(pp->scratch);
    if (pp->errFlag) errorWords().give(pp->errFlag);
    delete pp;
}

size_t smallPlanBytes(const void* h) {
    const PlanProgram* pp = reinterpret_cast<const PlanProgram*>(h);
    return pp ? pp->bytes + pp->scratch.bytes : 0;
}

// passes [first, last) of the plan; 0, a kernel's error code, or -1 when the launch failed
int smallPlanApply(void* h, float* re, float* im, int first, int last) {
    PlanProgram* pp = reinterpret_cast<PlanProgram*>(h);
    if (!launch(*pp, re, im, first, last, stream(), "applyPlanF32")) return -1;
    if (QG_CUDA(cudaStreamSynchronize(stream()), "applyPlanF32")) return -1;
    const int e = *reinterpret_cast<volatile int*>(pp->errFlag);
    if (e) {
        *pp->errFlag = 0;
        // a launch that gave up leaves the counters as they stood
        cudaMemsetAsync(pp->counters, 0, kCounterBytes, stream());
    }
    return e;
}

}  // namespace qg
