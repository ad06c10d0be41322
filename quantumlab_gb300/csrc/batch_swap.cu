// batch_swap.cu -- batched swap tests (QKMeans distances) in one persistent
// kernel, replayed through a CUDA graph.  No counterpart in the reference:
// QuantumLab runs one (2d+1)-qubit circuit at a time through the QuEST API
// (Code/QuantumLab/Circuit/Subroutine/QKMeans.cu:1158-1290,
// Code/QuantumLab/Circuit/Gates/SwapTest.cpp:15-68), each gate a launch.
//
// Circuit of one test (u, v of length 2^d, qubits: u = 0..d-1, v = d..2d-1,
// ancilla = 2d):   |0>|v>|u>  ->  H(anc)  ->  prod_i CSWAP(anc; u_i, v_i)
//                  ->  H(anc)  ->  P(anc = 0).
// The engine forms every amplitude of the anc = 0 half of the final state in
// registers and squares it: preparation + H(anc) gives phi(x, a, b) =
// u_a v_b / sqrt2 for both ancilla values (a = u-register index, b =
// v-register index); the d controlled swaps share the control and commute, so
// together they exchange the registers on the anc = 1 half, chi(1, a, b) =
// phi(1, b, a); H(anc) makes the amplitude omega(a, b) = (chi(0, a, b) +
// chi(1, a, b)) / sqrt2 = (u_a v_b + u_b v_a) / 2, and P(anc = 0) =
// sum_{a,b} |omega|^2.  (The powers of two are applied to the sum.)
//
// Nothing is stored between the gates: a state of 2^(2d+1) amplitudes written
// to and read back from device memory is what bounded an earlier form of this
// kernel (6.1 TB/s; 65,536 tests of d = 4..10 took 33.3 ms).  In registers an
// amplitude costs three FP32 operations (packed in twos) and a share of a
// shared-memory read, and the FP32 pipes bound it: 16,384 tests of d = 4..10
// 8.33 -> 0.24 ms, of which the FP32 operations take 0.16.  omega is symmetric, so above d = 6 the
// amplitudes with a and b in different blocks of 128 are formed once and
// counted twice.
//
// A lane owns NB values of b (u_b, v_b twice in a packed register each) and
// walks a four at a time, reading u_a, v_a as two broadcast 16-byte words;
// |omega|^2 is summed in FP32 over at most 8 terms per packed half and
// accumulator, the accumulators pairwise, and in FP64 above a unit of 16
// values of a.
//
// Scheduling: tests are sorted by size (largest first) and CTAs take the next
// item from a global ticket (atomicAdd), so uneven sizes balance.  An item is
// one test for the whole CTA (its units dealt to the warps) or, for small
// tests, one test per warp.
#include "qg_internal.h"
#include "quest_gb300.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <vector>

namespace qg {
namespace {

constexpr int kSwapThreads = 256;
constexpr int kSwapCtasPerSM = 4;        // the most CTAs per SM (launch bounds); the default
constexpr int kSmemAmps = 8192;          // default: a warp each for states of up to 2^13 amplitudes (d <= 6)
constexpr int kBlock = 128;              // values of b that a warp's lanes own together
constexpr int kUnit = 16;                // values of a per unit of work
constexpr int kMaxD = 10;

struct SwapJob {
    long long offA, offB;    // offsets of u and v in the vector pool
    int d;
    int out;                 // index into the result array
};

__device__ double blockSum(double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) red[w] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += red[k];
    __syncthreads();
    return t;
}

// two FP32 values in one register pair, and their packed operations
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float sum2(f32x2 a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
    return x + y;
}

// sum of (u_a v_b + u_b v_a)^2 over a = a0, a0 + 4 step, ... (count groups of
// four consecutive a, at most kUnit / 4) and the lane's NB values of b
template <int NB>
__device__ __forceinline__ float unitSum(const float* su, const float* sv, int a0, int count, int step,
                                         const f32x2 (&ub)[NB], const f32x2 (&vb)[NB]) {
    f32x2 acc[NB];
#pragma unroll
    for (int k = 0; k < NB; ++k) acc[k] = 0ull;
    for (int i = 0; i < count; ++i) {
        const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(su + a0 + 4 * i * step);
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(sv + a0 + 4 * i * step);
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            const f32x2 x = fma2(u.x, vb[k], mul2(ub[k], v.x)), y = fma2(u.y, vb[k], mul2(ub[k], v.y));
            acc[k] = fma2(y, y, fma2(x, x, acc[k]));
        }
    }
    float s[NB];
#pragma unroll
    for (int k = 0; k < NB; ++k) s[k] = sum2(acc[k]);
#pragma unroll
    for (int w = NB / 2; w > 0; w /= 2)
#pragma unroll
        for (int k = 0; k < w; ++k) s[k] += s[k + w];
    return s[0];
}

// the lane's values b0 + lane + 32 k
template <int NB>
__device__ __forceinline__ void loadB(const float* su, const float* sv, int b, f32x2 (&ub)[NB], f32x2 (&vb)[NB]) {
#pragma unroll
    for (int k = 0; k < NB; ++k) {
        ub[k] = pack2(su[b + 32 * k], su[b + 32 * k]);
        vb[k] = pack2(sv[b + 32 * k], sv[b + 32 * k]);
    }
}

// Units first, first + stride, ... of one test by one warp (D = 2^d values of
// a and b in su, sv); this lane's share of sum_{a,b} (u_a v_b + u_b v_a)^2.
template <int NB>
__device__ double squareUnits(const float* su, const float* sv, int D, int first, int stride, int lane) {
    f32x2 ub[NB], vb[NB];
    loadB<NB>(su, sv, lane, ub, vb);
    double total = 0.0;
    for (int a0 = first * kUnit; a0 < D; a0 += stride * kUnit) total += (double)unitSum<NB>(su, sv, a0, kUnit / 4, 1, ub, vb);
    return total;
}
__device__ __noinline__ double testUnits(const float* su, const float* sv, int d, int first, int stride, int lane) {
    const int D = 1 << d;
    if (d > 6) {
        // block j of b: the a below it in units counted twice, then the a of
        // the block itself; units are numbered through all blocks
        constexpr int kPerBlock = kBlock / kUnit, NB = kBlock / 32;
        f32x2 ub[NB], vb[NB];
        double total = 0.0;
        int unit = first, base = 0;                       // base: units of the blocks before j
        for (int j = 0; j < D / kBlock; ++j) {
            const int units = kPerBlock * (j + 1);
            if (unit < base + units) loadB<NB>(su, sv, j * kBlock + lane, ub, vb);
            for (; unit < base + units; unit += stride) {
                const float s = unitSum<NB>(su, sv, (unit - base) * kUnit, kUnit / 4, 1, ub, vb);
                total += (double)(unit - base < kPerBlock * j ? 2.f * s : s);
            }
            base += units;
        }
        return total;
    }
    if (d == 6) return squareUnits<2>(su, sv, D, first, stride, lane);
    if (d == 5) return squareUnits<1>(su, sv, D, first, stride, lane);
    if (first != 0) return 0.0;
    // D <= 16 values of b: the warp's 32 / D lane groups share the a (four at
    // a time; for D = 2 the upper half of each four is zero)
    f32x2 ub[1], vb[1];
    loadB<1>(su, sv, lane & (D - 1), ub, vb);
    const int group = lane >> d, groups = 32 >> d;
    const int fours = D > 4 ? D / 4 : 1;
    return group < fours ? (double)unitSum<1>(su, sv, 4 * group, (fours - group + groups - 1) / groups, groups, ub, vb) : 0.0;
}

__global__ void __launch_bounds__(kSwapThreads, kSwapCtasPerSM) kSwapTests(const float* __restrict__ pool,
                                                                           const SwapJob* __restrict__ jobs, int numJobs,
                                                                           int numBig, unsigned int* __restrict__ ticket,
                                                                           double* __restrict__ out) {
    constexpr int kWarps = kSwapThreads / 32, kSlice = (1 << kMaxD) / kWarps;   // a warp's own test: d <= 6
    static_assert(kSlice >= 64, "a warp's test must fit its slice");
    __shared__ __align__(16) float su[1 << kMaxD];
    __shared__ __align__(16) float sv[1 << kMaxD];
    __shared__ double red[kWarps];
    __shared__ int sItem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int numItems = numBig + (numJobs - numBig + kWarps - 1) / kWarps;
    for (;;) {
        if (threadIdx.x == 0) sItem = (int)atomicAdd(ticket, 1u);
        __syncthreads();
        const int item = sItem;
        __syncthreads();
        if (item >= numItems) break;
        if (item < numBig) {
            const SwapJob job = jobs[item];
            const int D = 1 << job.d;
            for (int i = threadIdx.x; i < D; i += kSwapThreads) {
                su[i] = pool[job.offA + i];
                sv[i] = pool[job.offB + i];
            }
            __syncthreads();
            const double p = blockSum(testUnits(su, sv, job.d, warp, kWarps, lane), red);
            if (threadIdx.x == 0) out[job.out] = 0.25 * p;
        } else {
            const int j = numBig + (item - numBig) * kWarps + warp;
            if (j < numJobs) {
                const SwapJob job = jobs[j];
                const int D = 1 << job.d;
                float* const wu = su + warp * kSlice;
                float* const wv = sv + warp * kSlice;
                for (int i = lane; i < D || i < 4; i += 32) {
                    wu[i] = i < D ? pool[job.offA + i] : 0.f;
                    wv[i] = i < D ? pool[job.offB + i] : 0.f;
                }
                __syncwarp();
                double p = testUnits(wu, wv, job.d, 0, 1, lane);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) p += __shfl_down_sync(0xffffffffu, p, o);
                if (lane == 0) out[job.out] = 0.25 * p;
            }
        }
        __syncthreads();                                  // su, sv are read no more
    }
}

struct SwapBatch {
    int numTests = 0;
    float* pool = nullptr;
    SwapJob* jobs = nullptr;
    unsigned int* ticket = nullptr;
    double* out = nullptr;
    int count[kMaxD + 1] = {};        // tests by d
    int ctasPerSM = kSwapCtasPerSM;   // tunable: 1 .. kSwapCtasPerSM
    int smemAmps = kSmemAmps;         // tunable: states of at most this many amplitudes take a warp, larger ones a CTA
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    double* hostOut = nullptr;        // pinned
};

void dropGraph(SwapBatch* b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
}

// the run's work on `st`: reset the ticket, the persistent kernel, results to
// pinned host memory
void queueSwaps(SwapBatch* b, cudaStream_t st) {
    int numBig = 0;                                       // the jobs are sorted, largest first
    for (int d = 1; d <= kMaxD; ++d)
        if (2ll << (2 * d) > b->smemAmps) numBig += b->count[d];
    cudaMemsetAsync(b->ticket, 0, sizeof(unsigned int), st);
    kSwapTests<<<numSMs() * b->ctasPerSM, kSwapThreads, 0, st>>>(b->pool, b->jobs, b->numTests, numBig, b->ticket, b->out);
    cudaMemcpyAsync(b->hostOut, b->out, b->numTests * sizeof(double), cudaMemcpyDeviceToHost, st);
}

// (re)capture the graph for the current parameters
bool captureSwaps(SwapBatch* b, const char* fn) {
    dropGraph(b);
    cudaStream_t cap = nullptr;
    if (QG_CUDA(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking), fn)) return false;
    bool ok = !QG_CUDA(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal), fn);
    if (ok) {
        queueSwaps(b, cap);
        ok = !QG_CUDA(cudaStreamEndCapture(cap, &b->graph), fn);
    }
    if (ok) ok = !QG_CUDA(cudaGraphInstantiate(&b->exec, b->graph, 0), fn);
    cudaStreamDestroy(cap);
    if (!ok) dropGraph(b);
    return ok;
}

void freeBatch(SwapBatch* b) {
    if (!b) return;
    cudaStreamSynchronize(stream());
    dropGraph(b);
    cudaFree(b->pool);
    cudaFree(b->jobs);
    cudaFree(b->ticket);
    cudaFree(b->out);
    cudaFreeHost(b->hostOut);
    delete b;
}

}  // namespace
}  // namespace qg

using qg::SwapBatch;
using qg::SwapJob;

extern "C" {

void* quest_gb300_swapTestBatchCreate(const double* vectors, const long long* offsets, const int* dimLog2,
                                      int numVectors, const int* idxA, const int* idxB, int numTests) {
    const char* fn = "quest_gb300_swapTestBatchCreate";
    if (!vectors || !offsets || !dimLog2 || !idxA || !idxB || numVectors < 1 || numTests < 1) {
        invalidQuESTInputError("Invalid swap-test batch arguments.", fn);
        return nullptr;
    }
    long long poolLen = 0;
    for (int i = 0; i < numVectors; ++i) {
        if (dimLog2[i] < 1 || dimLog2[i] > qg::kMaxD || offsets[i] < 0) {
            invalidQuESTInputError("Swap-test vectors must have length 2^d with 1 <= d <= 10.", fn);
            return nullptr;
        }
        poolLen = std::max(poolLen, offsets[i] + (1ll << dimLog2[i]));
    }
    std::vector<SwapJob> jobs(numTests);
    for (int t = 0; t < numTests; ++t) {
        const int a = idxA[t], b = idxB[t];
        if (a < 0 || a >= numVectors || b < 0 || b >= numVectors || dimLog2[a] != dimLog2[b]) {
            invalidQuESTInputError("Swap-test pair indices out of range or of unequal dimension.", fn);
            return nullptr;
        }
        jobs[t] = SwapJob{offsets[a], offsets[b], dimLog2[a], t};
    }
    // largest circuits first: dynamic scheduling then balances the tail
    std::stable_sort(jobs.begin(), jobs.end(), [](const SwapJob& x, const SwapJob& y) { return x.d > y.d; });
    SwapBatch* b = new SwapBatch();
    b->numTests = numTests;
    for (const SwapJob& j : jobs) ++b->count[j.d];
    std::vector<float> pool32(poolLen);
    for (long long i = 0; i < poolLen; ++i) pool32[i] = (float)vectors[i];
    cudaStream_t st = qg::stream();
    if (QG_CUDA(cudaMalloc(&b->pool, poolLen * sizeof(float)), fn) ||
        QG_CUDA(cudaMalloc(&b->jobs, numTests * sizeof(SwapJob)), fn) ||
        QG_CUDA(cudaMalloc(&b->ticket, sizeof(unsigned int)), fn) ||
        QG_CUDA(cudaMalloc(&b->out, numTests * sizeof(double)), fn) ||
        QG_CUDA(cudaMallocHost(&b->hostOut, numTests * sizeof(double)), fn)) {
        qg::freeBatch(b);
        return nullptr;
    }
    QG_CUDA(cudaMemcpyAsync(b->pool, pool32.data(), poolLen * sizeof(float), cudaMemcpyHostToDevice, st), fn);
    QG_CUDA(cudaMemcpyAsync(b->jobs, jobs.data(), numTests * sizeof(SwapJob), cudaMemcpyHostToDevice, st), fn);
    QG_CUDA(cudaStreamSynchronize(st), fn);
    if (!qg::captureSwaps(b, fn)) {
        qg::freeBatch(b);
        return nullptr;
    }
    return b;
}

// Time the batch with every pairing of CTAs per SM (2, 3, 4) and threshold
// (states of up to 2^9, 2^11 or 2^13 amplitudes, d <= 4, 5 or 6, take a warp
// each, larger ones a CTA), two runs each, keep the fastest and
// capture the graph again with it.  Writes the choice, its time and the time
// of the default (4 CTAs per SM, 2^13) in ms; returns 0 or -1.
int quest_gb300_swapTestBatchTune(void* batch, int* ctasPerSM, int* smemAmps, double* msBest, double* msDefault) {
    SwapBatch* b = reinterpret_cast<SwapBatch*>(batch);
    const char* fn = "quest_gb300_swapTestBatchTune";
    if (!b) return -1;
    cudaStream_t st = qg::stream();
    cudaEvent_t e0, e1;
    if (QG_CUDA(cudaEventCreate(&e0), fn) || QG_CUDA(cudaEventCreate(&e1), fn)) return -1;
    double best = -1, dflt = -1;
    int bestC = qg::kSwapCtasPerSM, bestS = qg::kSmemAmps;
    for (int c = 2; c <= qg::kSwapCtasPerSM; ++c)
        for (int sm : {512, 2048, 8192}) {
            b->ctasPerSM = c;
            b->smemAmps = sm;
            qg::queueSwaps(b, st);                    // warm-up
            cudaEventRecord(e0, st);
            for (int r = 0; r < 2; ++r) qg::queueSwaps(b, st);
            cudaEventRecord(e1, st);
            if (QG_CUDA(cudaEventSynchronize(e1), fn)) return -1;
            float ms = 0;
            cudaEventElapsedTime(&ms, e0, e1);
            const double per = ms / 2.0;
            if (c == qg::kSwapCtasPerSM && sm == qg::kSmemAmps) dflt = per;
            if (best < 0 || per < best) {
                best = per;
                bestC = c;
                bestS = sm;
            }
        }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    b->ctasPerSM = bestC;
    b->smemAmps = bestS;
    if (!qg::captureSwaps(b, fn)) return -1;
    if (ctasPerSM) *ctasPerSM = bestC;
    if (smemAmps) *smemAmps = bestS;
    if (msBest) *msBest = best;
    if (msDefault) *msDefault = dflt;
    return 0;
}

// Replay the batch's graph on the library stream and write P(anc = 0) of
// every test (in the caller's order) to p0Out (host memory).
int quest_gb300_swapTestBatchRun(void* batch, double* p0Out) {
    SwapBatch* b = reinterpret_cast<SwapBatch*>(batch);
    const char* fn = "quest_gb300_swapTestBatchRun";
    if (!b) return -1;
    cudaStream_t st = qg::stream();
    if (QG_CUDA(cudaGraphLaunch(b->exec, st), fn)) return -1;
    qg::g_launches.fetch_add(1);
    if (QG_CUDA(cudaStreamSynchronize(st), fn)) return -1;
    if (p0Out) std::memcpy(p0Out, b->hostOut, b->numTests * sizeof(double));
    return 0;
}

void quest_gb300_swapTestBatchDestroy(void* batch) { qg::freeBatch(reinterpret_cast<SwapBatch*>(batch)); }

}  // extern "C"
