// launch_util.h -- host helpers of the kernel launchers.
#pragma once

#include <cuda_runtime.h>

#include <atomic>

namespace qld {

// Allow `kern` `bytes` of dynamic shared memory, once per device: `done` is
// the kernel's own static, one bit per device (devices past 63 ask each time).
template <typename Kernel>
cudaError_t allow_smem(Kernel kern, int bytes, std::atomic<unsigned long long> &done) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return e;
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
