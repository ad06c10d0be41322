// chain_launch.cuh -- kernels that follow one another on the library stream,
// launched so that the next grid's blocks start on SMs as the previous grid
// leaves them (programmatic dependent launch).
//
// A small gate is all launch latency: one after the other, plain launches of
// kernels that run about 2 us come 4.1 us apart, in steps of 2.05 us (4.1,
// 6.2, 8.3, 10.3).  A kernel launched with chain() calls chainStart() before
// it touches memory: it lets its own successor start, then waits until the
// grids before it have ended and their writes are visible.  Every access of
// global memory stands behind that wait, so the order of the stream is kept;
// work that is launched plainly before or after orders as always.
// A chained kernel's pointers are not __restrict__ and it does not use __ldg:
// either lets the compiler read through the non-coherent path, which holds
// only for data that stays unchanged while the kernel is resident, or move a
// load to before the wait.  Both kinds of block are resident while the grid
// before still writes (phase tables, pass products, operand images, the state).
// From gate to gate, 16 qubits 4.1 -> 2.5 us, 20 qubits: compactUnitary 10.4
// -> 8.5, rotations 8.3 -> 6.2, phases 6.2 -> 4.2; a 9-qubit circuit of 70
// calls 285 -> 164 us, now bound by the calls.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <mutex>
#include <utility>

namespace qg {

int numSMs();

__device__ __forceinline__ void chainStart() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A grid of a few blocks an SM starts while the grid before holds its places,
// and its blocks then crowd where places are free first: 256 blocks (18 qubits)
// of a gate bound by the FP64 pipe took 13.2 us, launched plainly 8.2.  Shared
// memory that is not used keeps an SM to the even share.
constexpr size_t kEvenShareBytes = 200 * 1024;
inline size_t evenShare(unsigned blocks) {
    const unsigned sms = (unsigned)numSMs(), each = (blocks + sms - 1) / sms;
    // each + 1 such blocks do not fit 228 KB, and one leaves 27 KB for a kernel's own
    return 2 * blocks > sms && each <= 4 ? kEvenShareBytes / each : 0;
}
// Let a kernel's launches take up to `most` bytes of dynamic shared memory.  The
// limit belongs to the process, and to set it while another thread launches the
// kernel may fail that launch (or crash in the driver).  So it is set once, to
// the most that any launch takes, before the kernel's first launch.
template <auto kernel>
inline cudaError_t allowShared(size_t most) {
    static std::mutex mutex;
    static std::atomic<bool> set{false};
    if (set.load(std::memory_order_acquire)) return cudaSuccess;
    std::lock_guard<std::mutex> lk(mutex);
    if (set.load(std::memory_order_relaxed)) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e == cudaSuccess) set.store(true, std::memory_order_release);
    return e;
}

// `cluster`: blocks to a thread-block cluster (of consecutive blocks in x)
template <class... Params, class... Args>
inline void launchChained(unsigned cluster, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                          Args&&... args) {
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    (void)cudaLaunchKernelEx(&cfg, kernel, Params(std::forward<Args>(args))...);     // its error: launchFailed
}
// A kernel without shared memory of its own takes the even share's.
template <auto kernel, class... Args>
inline void chain(dim3 grid, dim3 block, cudaStream_t st, Args&&... args) {
    const bool allowed = allowShared<kernel>(kEvenShareBytes) == cudaSuccess;
    if (!allowed) (void)cudaGetLastError();          // it runs without the share
    launchChained(1, kernel, grid, block, allowed ? evenShare(grid.x * grid.y) : 0, st, std::forward<Args>(args)...);
}
// One with `smem` bytes, which allowShared has been asked for.
template <auto kernel, class... Args>
inline void chainShared(unsigned cluster, dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    launchChained(cluster, kernel, grid, block, smem, st, std::forward<Args>(args)...);
}

}  // namespace qg
