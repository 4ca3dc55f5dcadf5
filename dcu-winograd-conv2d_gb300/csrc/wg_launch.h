// Kernel launches with programmatic dependent launch (PDL): each kernel of a
// convolution may be scheduled while the kernel before it on the stream is
// still finishing, runs its prologue (barrier set-up, descriptor prefetch),
// and waits in griddepcontrol.wait for the earlier grid's completion and
// memory flush before it touches any tensor.  Every kernel launched this way
// starts with that wait, so results and ordering are those of plain stream
// launches; only the launch gap and prologue overlap.  WG_CONV2D_PDL=0 turns
// it off (plain launches).
#pragma once
#include <atomic>
#include <cstdlib>
#include <mutex>
#include <utility>

#include <cuda_runtime.h>

namespace wg {

inline bool pdl_enabled() {
    static const bool on = [] {
        const char* v = std::getenv("WG_CONV2D_PDL");
        return !(v && v[0] == '0');
    }();
    return on;
}

// Raises the kernel's dynamic shared memory limit to `bytes` on the current
// device, once (the limit stays until the process ends): asking the runtime on
// every launch cost 0.3-0.4 us of host time (a call of one kernel 3.58 -> 3.18 us
// to submit, of three 7.6 -> 6.7).  Limit and cached value are raised under one
// lock and never lowered: of two threads that raise a kernel's limit at once, by
// unlike sizes, neither may leave a cached value above the limit in force.
template <auto Kernel>
cudaError_t allow_smem(int bytes) {
    constexpr int kDevices = 64;
    static std::atomic<int> allowed[kDevices] = {};
    static std::mutex raising;
    int dev = 0;
    if (cudaError_t e = cudaGetDevice(&dev); e != cudaSuccess) return e;
    if (dev < kDevices && allowed[dev].load(std::memory_order_acquire) >= bytes) return cudaSuccess;
    std::lock_guard<std::mutex> lock(raising);
    if (dev < kDevices && allowed[dev].load(std::memory_order_relaxed) >= bytes) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && dev < kDevices) allowed[dev].store(bytes, std::memory_order_release);
    return e;
}

template <class... KArgs, class... Args>
cudaError_t launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

// The same for a kernel of CTA pairs (clusters of two): `pairs` clusters.
template <class... KArgs, class... Args>
cudaError_t launch_pairs(void (*kern)(KArgs...), int pairs, int threads, size_t smem, cudaStream_t s, const Args&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

}  // namespace wg
