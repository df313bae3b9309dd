// Per-device facts the kernel launchers size their grids by, looked up once
// per device ordinal (a process may drive more than one GPU, one after the
// other, and GPUs of one machine need not have the same SM count).
#pragma once

#include <cuda_runtime.h>

#include <atomic>

namespace gbdev {

// Programmatic stream serialisation: a kernel launched by launchAfter() may start as soon as every CTA of the kernel
// before it has called nextMayLaunch() or ended.  waitForKernelBefore() waits until that kernel (and what it waited
// for) has ended and its writes are visible; every thread of a kernel so launched calls it, before it reads anything
// that kernel writes, and before it ends.
__device__ __forceinline__ void nextMayLaunch() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void waitForKernelBefore() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... Params, typename... Args>
inline cudaError_t launchAfterShared(void (*kernel)(Params...), unsigned blocks, unsigned threads, size_t shared,
                                     cudaStream_t s, Args... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(blocks);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = shared;
    c.stream = s;
    c.attrs = &attr;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, Params(args)...);
}
template <typename... Params, typename... Args>
inline cudaError_t launchAfter(void (*kernel)(Params...), unsigned blocks, unsigned threads, cudaStream_t s,
                               Args... args) {
    return launchAfterShared(kernel, blocks, threads, 0, s, args...);
}

constexpr int MAX_DEVICES = 64;

// the current device's ordinal, or -1
inline int current() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return -1;
    return dev;
}

// SM count of the current device (152 on GB300 if the query fails)
inline int smCount() {
    static std::atomic<int> cache[MAX_DEVICES];
    const int dev = current();
    if (dev < 0) return 152;
    int n = cache[dev].load(std::memory_order_relaxed);
    if (n <= 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 152;
        cache[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

// CTAs of `kernel` (threads per CTA, dynamic shared memory) that are resident
// on one SM of the current device; the dynamic shared memory limit is raised
// first where it exceeds the default.  Cached per (device, cache) slot:
// one `cache` array per kernel/configuration.
template <typename K>
int residentCtas(std::atomic<int> (&cache)[MAX_DEVICES], K kernel, int threads, size_t smem) {
    const int dev = current();
    if (dev < 0) return 1;
    int occ = cache[dev].load(std::memory_order_relaxed);
    if (occ <= 0) {
        if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem) != cudaSuccess || occ < 1)
            occ = 1;
        cache[dev].store(occ, std::memory_order_relaxed);
    }
    return occ;
}

}  // namespace gbdev
