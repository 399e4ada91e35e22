// Host-side helpers shared by the translation units of libcdssm_b200.so.
#pragma once
#include "../../include/cdssm_b200.h"
#include "cdssm_math.cuh"
#include <atomic>

namespace cdssm {

// CUDA error of the last failed call on this host thread (read by cdssm_b200_last_cuda_error).
int& last_cuda_error_ref();

inline int check_cuda(cudaError_t e) {
    if (e == cudaSuccess) return CDSSM_OK;
    last_cuda_error_ref() = (int)e;
    return CDSSM_ERR_CUDA;
}
// Kernels this library has launched in this process (cdssm_b200_launch_count).
std::atomic<long long>& launch_count_ref();
inline int counted(int rc) {
    if (rc == CDSSM_OK) launch_count_ref().fetch_add(1, std::memory_order_relaxed);
    return rc;
}
inline int check_launch() { return counted(check_cuda(cudaGetLastError())); }

// Programmatic dependent launch: the kernel may start while its predecessor in the stream drains; it must not touch
// anything a predecessor writes (nor write anything a predecessor reads) before grid_dependency_wait().
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
inline int launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return counted(check_cuda(cudaLaunchKernelEx(&cfg, kernel, P(args)...)));
}

// Multiprocessors of the current device.
inline int sm_count(int& sms) {
    int dev = 0;
    if (int rc = check_cuda(cudaGetDevice(&dev))) return rc;
    return check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
}

// Opts a kernel in to `bytes` of dynamic shared memory, once per kernel (Tag) and device.
template <typename Tag>
inline int allow_smem(const void* kernel, size_t bytes) {
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    if (int rc = check_cuda(cudaGetDevice(&dev))) return rc;
    const uint64_t bit = 1ull << (dev & 63);
    if (dev < 64 && (done.load(std::memory_order_relaxed) & bit)) return CDSSM_OK;
    if (int rc = check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes))) return rc;
    done.fetch_or(bit, std::memory_order_relaxed);
    return CDSSM_OK;
}

}  // namespace cdssm
