// Host-side plumbing shared by the translation units of libkrr_gb300.so:
// status codes, the per-thread last-error text and CUDA error mapping.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string>

#include "../../include/krr_gb300.h"
#include "per_device.h"

namespace krr {

void set_last_error(const std::string &msg);
int fail(int status, const char *fmt, ...);

inline int cuda_status(cudaError_t e, const char *what, const char *file, int line) {
    if (e == cudaSuccess) return KRR_OK;
    return fail(e == cudaErrorMemoryAllocation ? KRR_ERR_OUT_OF_MEMORY : KRR_ERR_CUDA,
                "%s failed at %s:%d: %s", what, file, line, cudaGetErrorString(e));
}

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

// Device-side error flags (set by kernels instead of trapping).
enum DeviceError : uint32_t {
    kErrStackOverflow = 1u << 0,
    kErrQueueOverflow = 1u << 1,
    kErrLoopLimit = 1u << 2,
    kErrBadInput = 1u << 3,
};

// Launches a kernel that may be brought up while the one before it on the
// stream still runs; the kernel starts with stream_order() (kmath.cuh), which
// waits for that one's end and its writes.  Between short dependent kernels
// this hides the launch itself.  After anything that is not such a kernel
// (copies, memsets, other launches) and for anything after it, the order is
// the stream's as always.
// The kernel's blocks may be resident while the one before it writes, so what
// that one writes is not read-only for the kernel's life: it is read through
// pointers that are not `const __restrict__`, and never by __ldg.  The
// compiler may move those loads before stream_order() (a memory clobber does
// not hold loads that it takes to be invariant) and serve them from the
// read-only path.  Both are fine for what has been written before the kernel
// before: the tree, the scene, the frame's views and constants.
template <typename... P, typename... A>
inline cudaError_t launch_ordered(void (*kernel)(P...), int grid, int block, cudaStream_t s, A &&...args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Raises a kernel's dynamic shared-memory limit, which belongs to the kernel
// on one device: `done` is that kernel's own.
template <typename... P>
inline cudaError_t allow_shared(OncePerDevice &done, void (*kernel)(P...), size_t bytes) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    return (cudaError_t)done(dev, [&] {
        return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    });
}

}  // namespace krr

#define KRR_CUDA(call)                                                              \
    do {                                                                            \
        cudaError_t _e = (call);                                                    \
        if (_e != cudaSuccess) return ::krr::cuda_status(_e, #call, __FILE__, __LINE__); \
    } while (0)

#define KRR_TRY(call)                  \
    do {                               \
        int _s = (call);               \
        if (_s != KRR_OK) return _s;   \
    } while (0)

#define KRR_CHECK_ARG(cond, msg)                                                   \
    do {                                                                           \
        if (!(cond)) return ::krr::fail(KRR_ERR_INVALID_ARGUMENT, "%s", msg);      \
    } while (0)
