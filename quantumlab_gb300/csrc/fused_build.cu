// fused_build.cu -- the operands of a plan's passes formed on the device
// (sm_103a).  No counterpart in the reference.
//
// A capture flush plans a circuit it runs once or with other angles each time.
// Forming its pass products and operand images on host threads, copying them
// and allocating for them took 1.6 ms of the 2.2 ms of a 20-qubit, 8-layer
// flush, whose 26 passes take 0.3 ms.  Here the host sends the gates (some 70
// KB); one kernel multiplies each pass's gates in FP64 (eight blocks a pass,
// each its share of the columns, which a product from the left keeps apart),
// another writes the operand forms, entry by entry as the host code does.
// The whole case (316 calls, flush, total probability): 2.24 ms -> 0.75 ms.
#include "chain_launch.cuh"
#include "fused_build.h"
#include "qg_internal.h"

#include <algorithm>
#include <cstring>
#include <cuda_fp16.h>

namespace qg {
namespace {

constexpr int kThreads = 256;
constexpr int kSlices = 8;               // blocks a pass: products (columns), images (entries)
constexpr int kMaxGateQubits = 3;
constexpr int kF16XExp = 14, kF16GMaxExp = 14;     // as in fused_tc.cu

struct DevGate {
    int q;                               // qubits
    int pos[kMaxGateQubits];             // their bits in the pass's index, in the gate's bit order
    uint32_t m;                          // first entry of its matrix
};
struct DevPass {
    int k, gate, gates;
    int smallMask;
    uint64_t product;                    // entries to its product
    uint64_t full, bf16, compact, f16, small;
};

// y + g x; a call, so that an entry that is zero takes a branch: predicated
// off, its FP64 instructions would still take their slots
__device__ __noinline__ double2 addProduct(double2 y, double2 g, double2 x) {
    return make_double2(y.x + (g.x * x.x - g.y * x.y), y.y + (g.x * x.y + g.y * x.x));
}
// a gate on Q qubits from the left, on the block's W columns of the product
template <int Q>
__device__ __forceinline__ void applyGate(double2* m, const double2* u, const DevGate& dg, int D, int W) {
    constexpr int G = 1 << Q;
    int low[Q];                          // its bits, ascending
#pragma unroll
    for (int t = 0; t < Q; ++t) low[t] = dg.pos[t];
#pragma unroll
    for (int a = 0; a < Q; ++a)
#pragma unroll
        for (int b = a + 1; b < Q; ++b)
            if (low[b] < low[a]) {
                const int t = low[a];
                low[a] = low[b];
                low[b] = t;
            }
    for (int i = threadIdx.x; i < (D >> Q) * W; i += kThreads) {
        int row = i / W;
        const int c = i % W;
#pragma unroll
        for (int t = 0; t < Q; ++t) row = ((row >> low[t]) << (low[t] + 1)) | (row & ((1 << low[t]) - 1));
        double2 x[G];
        int at[G];
#pragma unroll
        for (int e = 0; e < G; ++e) {
            int r = row;
#pragma unroll
            for (int t = 0; t < Q; ++t) r |= (e >> t & 1) << dg.pos[t];
            at[e] = r * W + c;
            x[e] = m[at[e]];
        }
#pragma unroll
        for (int a = 0; a < G; ++a) {
            double2 y = make_double2(0.0, 0.0);
#pragma unroll
            for (int e = 0; e < G; ++e) {
                const double2 g = u[a * G + e];
                if (Q < 2) {
                    y.x += g.x * x[e].x - g.y * x[e].y;
                    y.y += g.x * x[e].y + g.y * x[e].x;
                } else if (g.x != 0.0 || g.y != 0.0) {
                    y = addProduct(y, g, x[e]);
                }
            }
            m[at[a]] = y;
        }
    }
}

// products: D x D entries a pass, row-major
__global__ void __launch_bounds__(kThreads) kProducts(const DevPass* passes, const DevGate* gates,
                                                      const double2* entries, double2* products, unsigned long long* largest) {
    constexpr int kMaxEntries = 1 << (2 * kMaxGateQubits);
    __shared__ double2 m[64 * 64 / kSlices];
    __shared__ double2 entry[2][kMaxEntries];      // this gate's, the next one's
    __shared__ DevGate gate[3];                    // this one, the next two
    chainStart();
    const int tid = threadIdx.x;
    const DevPass p = passes[blockIdx.x];
    const int D = 1 << p.k, W = max(1, D / kSlices), c0 = blockIdx.y * W;
    if (c0 >= D) return;
    for (int i = tid; i < D * W; i += kThreads) m[i] = make_double2(i / W == c0 + i % W ? 1.0 : 0.0, 0.0);
    if (tid < 2 && tid < p.gates) gate[tid] = gates[p.gate + tid];
    __syncthreads();
    if (p.gates > 0 && tid < 1 << (2 * gate[0].q)) entry[0][tid] = entries[gate[0].m + tid];
    for (int g = 0; g < p.gates; ++g) {
        __syncthreads();
        const DevGate dg = gate[g % 3];
        const double2* u = entry[g & 1];
        // the next gate's entries, the one after's description
        if (g + 1 < p.gates && tid < 1 << (2 * gate[(g + 1) % 3].q)) entry[(g + 1) & 1][tid] = entries[gate[(g + 1) % 3].m + tid];
        if (g + 2 < p.gates && tid == kThreads - 1) gate[(g + 2) % 3] = gates[p.gate + g + 2];
        if (dg.q == 1) applyGate<1>(m, u, dg, D, W);
        else if (dg.q == 2) applyGate<2>(m, u, dg, D, W);
        else applyGate<3>(m, u, dg, D, W);
    }
    __syncthreads();
    unsigned long long big = 0;
    for (int i = threadIdx.x; i < D * W; i += kThreads) {
        const double2 v = m[i];
        products[p.product + (i / W) * D + c0 + i % W] = v;
        const unsigned long long a = __double_as_longlong(fabs(v.x)), b = __double_as_longlong(fabs(v.y));
        big = max(big, max(a, b));
    }
    if (p.f16 != ~0ull) atomicMax(largest + blockIdx.x, big);      // bits of nonnegative doubles order as numbers
}

__device__ __forceinline__ float tf32(float x) {
    uint32_t u = __float_as_uint(x);
    if ((u & 0x7F800000u) != 0x7F800000u) u = (u + 0x1000u) & 0xFFFFE000u;
    return __uint_as_float(u);
}
__device__ __forceinline__ uint16_t bf16(float x) {
    uint32_t u = __float_as_uint(x);
    u += 0x7FFFu + ((u >> 16) & 1u);
    return (uint16_t)(u >> 16);
}
__device__ __forceinline__ size_t kMajor(int r, int j, int K) {        // packKMajor, in floats
    return (size_t)(r / 8) * (K / 4) * 32 + (size_t)(j / 4) * 32 + (r % 8) * 4 + j % 4;
}

__global__ void __launch_bounds__(kThreads) kImages(const DevPass* passes, const double2* products,
                                                    const unsigned long long* largest, float* out) {
    chainStart();
    const DevPass p = passes[blockIdx.x];
    const int D = 1 << p.k, N = 2 * D;
    const double2* M = products + p.product;
    const int first = blockIdx.y * kThreads + threadIdx.x, step = kSlices * kThreads;
    // entry (r, j) of the real form [[Re, -Im], [Im, Re]]
    auto real = [&](int r, int j) {
        const double2 g = M[(r % D) * D + j % D];
        return (r < D) == (j < D) ? g.x : r < D ? -g.y : g.y;
    };
    // row r of the compact form [-Im; Re; Im] (6 qubits) is (r, D + j) or (r - D, j)
    auto compactEntry = [&](int r, int j) { return r < D ? real(r, D + j) : real(r - D, j); };
    if (p.small != ~0ull) {
        auto own = [&](int i) {
            int v = 0;
            for (int b = 0, o = 0; b < 6; ++b)
                if (p.smallMask >> b & 1) v |= (i >> b & 1) << o++;
            return v;
        };
        for (int e = first; e < 4096; e += step) {
            const int j = e / 64, r = e % 64;
            double2 v = make_double2(0.0, 0.0);
            if (((r ^ j) & ~p.smallMask & 63) == 0) v = M[own(r) * D + own(j)];
            out[p.small + e] = (float)v.x;
            out[p.small + 4096 + e] = (float)v.y;
        }
    }
    if (p.full != ~0ull)
        for (int e = first; e < N * N; e += step) {
            const int r = e / N, j = e % N;
            const double v = real(r, j);
            const float h = tf32((float)v);
            out[p.full + kMajor(r, j, N)] = h;
            out[p.full + (size_t)N * N + kMajor(r, j, N)] = tf32((float)(v - (double)h));
        }
    if (p.compact != ~0ull)
        for (int e = first; e < 3 * D * D; e += step) {
            const int r = e / D, j = e % D;
            const double v = compactEntry(r, j);
            const float h = tf32((float)v);
            out[p.compact + kMajor(r, j, D)] = h;
            out[p.compact + (size_t)3 * D * D + kMajor(r, j, D)] = tf32((float)(v - (double)h));
        }
    const int rows = p.k == 6 ? 3 * D : N, cols = p.k == 6 ? D : N;
    const size_t entries = (size_t)rows * cols;
    auto core = [&](int r, int j) { return (size_t)(r / 8) * (cols / 8) * 64 + (size_t)(j / 8) * 64 + (r % 8) * 8 + j % 8; };
    if (p.bf16 != ~0ull) {
        uint16_t* o = reinterpret_cast<uint16_t*>(out + p.bf16);
        for (int e = first; e < (int)entries; e += step) {
            const int r = e / cols, j = e % cols;
            const double v = p.k == 6 ? compactEntry(r, j) : real(r, j);
            const uint16_t h = bf16((float)v);
            const double r1 = v - (double)__uint_as_float((uint32_t)h << 16);
            const uint16_t l = bf16((float)r1);
            o[core(r, j)] = h;
            o[entries + core(r, j)] = l;
            o[2 * entries + core(r, j)] = bf16((float)(r1 - (double)__uint_as_float((uint32_t)l << 16)));
        }
    }
    if (p.f16 != ~0ull) {
        const double mx = __longlong_as_double((long long)largest[blockIdx.x]);
        int sc = 24;
        if (mx > 0.0) {
            int e2 = 0;
            frexp(mx, &e2);
            sc = min(24, max(-24, kF16GMaxExp - e2));
        }
        uint16_t* o = reinterpret_cast<uint16_t*>(out + p.f16);
        for (int e = first; e < (int)entries; e += step) {
            const int r = e / cols, j = e % cols;
            const double v = scalbn(p.k == 6 ? compactEntry(r, j) : real(r, j), sc);
            const __half h = __double2half(v);
            o[core(r, j)] = __half_as_ushort(h);
            o[entries + core(r, j)] = __half_as_ushort(__double2half(v - (double)__half2float(h)));
        }
        if (first < 4) out[p.f16 + entries + first] = first == 0 ? scalbnf(1.f, -(kF16XExp + sc)) : 0.f;
    }
}

}  // namespace

void freeBuildScratch(BuildScratch& s) {
    s.source.release();
    if (s.device) cudaFree(s.device);
    s.device = nullptr;
    s.bytes = 0;
}

bool buildsOnDevice(const FusedPlan& plan, const FusedPass& pass, const std::vector<int>& members) {
    if (!pass.controls.empty() || pass.targets.size() > 6) return false;
    for (int i : members)
        if (plan.gates[i].qubits.size() > (size_t)kMaxGateQubits) return false;
    return true;
}

bool queueBuild(const FusedPlan& plan, const std::vector<int>& which, const std::vector<BuildOutput>& outputs, float* out,
                BuildScratch& scratch, cudaStream_t st, const char* caller) {
    if (which.empty()) return true;
    std::vector<DevPass> passes;
    std::vector<DevGate> gates;
    std::vector<cplx> entries;
    size_t product = 0;
    for (size_t w = 0; w < which.size(); ++w) {
        const FusedPass& pass = plan.passes[which[w]];
        const BuildOutput& o = outputs[w];
        DevPass d{};
        d.k = (int)pass.targets.size();
        d.gate = (int)gates.size();
        d.smallMask = o.smallMask;
        d.product = product;
        product += (size_t)1 << (2 * d.k);
        d.full = o.full; d.bf16 = o.bf16; d.compact = o.compact; d.f16 = o.f16; d.small = o.small;
        for (int i : plan.passMembers[which[w]]) {
            const FusedGate& g = plan.gates[i];
            DevGate dg{};
            dg.q = (int)g.qubits.size();
            for (int t = 0; t < dg.q; ++t)
                dg.pos[t] = (int)(std::lower_bound(pass.targets.begin(), pass.targets.end(), g.qubits[t]) - pass.targets.begin());
            dg.m = (uint32_t)entries.size();
            entries.insert(entries.end(), g.m.begin(), g.m.end());
            gates.push_back(dg);
        }
        d.gates = (int)gates.size() - d.gate;
        passes.push_back(d);
    }
    // one upload: entries, passes, gates; behind it the products and maxima
    auto up16 = [](size_t b) { return (b + 15) / 16 * 16; };
    const size_t eAt = 0, pAt = up16(entries.size() * sizeof(cplx)), gAt = pAt + up16(passes.size() * sizeof(DevPass));
    const size_t mAt = gAt + up16(gates.size() * sizeof(DevGate)), upload = mAt + up16(passes.size() * 8);
    const size_t need = upload + product * sizeof(double2);
    if (scratch.bytes < need) {
        freeBuildScratch(scratch);
        if (QG_CUDA(cudaMalloc(&scratch.device, need), caller)) return false;
        scratch.bytes = need;
    }
    char* host = scratch.source.open(upload, caller);    // (maxima start at 0)
    if (!host) return false;
    memcpy(host + eAt, entries.data(), entries.size() * sizeof(cplx));
    memcpy(host + pAt, passes.data(), passes.size() * sizeof(DevPass));
    memcpy(host + gAt, gates.data(), gates.size() * sizeof(DevGate));
    char* dev = reinterpret_cast<char*>(scratch.device);
    if (!scratch.source.copy(dev, st, caller)) return false;
    const DevPass* dp = reinterpret_cast<const DevPass*>(dev + pAt);
    double2* products = reinterpret_cast<double2*>(dev + upload);
    unsigned long long* largest = reinterpret_cast<unsigned long long*>(dev + mAt);
    const dim3 grid((unsigned)passes.size(), kSlices);
    chain<kProducts>(grid, kThreads, st, dp, reinterpret_cast<const DevGate*>(dev + gAt),
          reinterpret_cast<const double2*>(dev + eAt), products, largest);
    if (launchFailed(caller)) return false;
    chain<kImages>(grid, kThreads, st, dp, products, largest, out);
    return !launchFailed(caller);
}

}  // namespace qg
