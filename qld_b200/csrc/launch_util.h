// launch_util.h -- host helpers of the kernel launchers.
#pragma once

#include <cuda_runtime.h>

#include <atomic>

namespace qld {

// Counts the contexts made so far (qld_cuda_init).  A kernel's attributes last
// as long as the device's own context, which cudaDeviceReset ends; whatever
// launches after that does so from a context made later.
extern std::atomic<unsigned> g_context_epoch;

// Allow `kern` `bytes` of dynamic shared memory, once per device since the last
// context was made: `done` is the kernel's own static, that epoch and a bit per
// device (devices past 31 ask each time).
template <typename Kernel>
cudaError_t allow_smem(Kernel kern, int bytes, std::atomic<unsigned long long> &done) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long epoch =
        (unsigned long long)g_context_epoch.load(std::memory_order_acquire) << 32;
    const unsigned long long bit = dev < 32 ? 1ull << dev : 0ull, devices = 0xFFFFFFFFull;
    unsigned long long known = done.load(std::memory_order_acquire);
    if ((known & ~devices) == epoch && (known & bit)) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    while (!done.compare_exchange_weak(
        known, (known & ~devices) == epoch ? known | bit : epoch | bit, std::memory_order_release,
        std::memory_order_relaxed)) {}
    return cudaSuccess;
}

// Attribute: the kernel may start (its set-up, up to griddep_wait) while the
// kernel before it in the stream is still finishing.
inline cudaLaunchAttribute overlap_attr() {
    cudaLaunchAttribute a = {};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    return a;
}

}  // namespace qld
