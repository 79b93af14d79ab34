// wlc_attr.h -- kernel attributes, which CUDA keeps per device.
//
// cudaFuncSetAttribute(MaxDynamicSharedMemorySize) applies to the device
// that is current when it is called.  A process that launches on several
// devices (one context per device, or the allocation-free step on each
// GPU) must set it once per (kernel, device); a single process-wide flag
// would leave every device but the first at the 48 KB default and make
// their large-shared-memory launches fail.
#pragma once
#include <cuda_runtime.h>

#include <mutex>
#include <set>
#include <utility>

namespace wlc {

// Raise the dynamic shared-memory limit of kernel `fn` to `bytes` on the
// current device, once per (kernel, device).  Thread-safe; returns the
// error of cudaGetDevice / cudaFuncSetAttribute (nothing is recorded on
// failure, so a later call retries).
inline cudaError_t smem_attr_once(const void* fn, int bytes) {
    static std::mutex mu;
    static std::set<std::pair<const void*, int>> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    if (done.count({fn, dev})) return cudaSuccess;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) done.insert({fn, dev});
    return e;
}

template <typename K> inline cudaError_t smem_attr_once(K* fn, int bytes) {
    return smem_attr_once(reinterpret_cast<const void*>(fn), bytes);
}

// Launch of a kernel that begins with dep_wait() below: with `chain` it may be
// put in place while the kernel before it on the stream finishes (programmatic
// dependent launch), which takes the launch latency between the passes of a
// contour step off their chain.  chained_step: where that was faster at every
// degree.  Both sweeps and the density, chained against not, 17 pairs of grid
// and degree in FP32 and 15 in FP64: FP32 16^3 .. 40^3 (L = 1 .. 12) 0.75-0.99
// of the time, 48^3 0.88-1.01; FP64 8^3 .. 24^3 (L = 1 .. 10) 0.85-1.00.  Above,
// CTAs put in place early hold shared memory that the other sweep's kernels
// could use: FP64 32^3, L = 6 1.03, FP32 64^3, L = 10 1.01 (lower degrees there
// would gain 2-9 %).
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr bool chained_step(int N, int tsize, bool batched) { return !batched && N <= (tsize == 4 ? 48 : 24); }
template <typename... P, typename... A>
inline cudaError_t launch_chained(bool chain, void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t st,
                                  A... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = chain ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
#ifdef __CUDACC__
// every kernel before this one on the stream has finished and its writes are visible
template <bool CHAINED> __device__ __forceinline__ void dep_wait() {
    if constexpr (CHAINED) asm volatile("griddepcontrol.wait;" ::: "memory");
}
// the next kernel on the stream may be put in place once every CTA has come here
template <bool CHAINED> __device__ __forceinline__ void dep_next() {
    if constexpr (CHAINED) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif

}  // namespace wlc
