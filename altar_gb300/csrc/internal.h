// Host-side helpers shared by the C-ABI translation units.
#pragma once
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdio.h>

#include "../../include/altar_gb300.h"

namespace ag {

// records the calling thread's last error message and returns `code`
int set_error(int code, const char* fmt, ...);

// translate a CUDA runtime status: AG_OK or AG_ERR_CUDA with the message recorded
int cuda_status(cudaError_t e, const char* where);

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<size_t>(p) % a) == 0; }

// Launch behind the kernel before it on the stream without waiting for that one's last CTA to leave
// first (programmatic dependent launch).  The kernel's first statement is after_previous(), so it
// touches memory only when its predecessor has ended; what it saves is the gap, ~2 µs per launch of
// a chain of short kernels: linear model (4 kernels, 16,384 chains) 107 -> 98 µs, surrogate
// prediction (8) 158 -> 141, a stage's schedule, covariance and resampling (8) 275 -> 261, training
// (8 per batch) 769 -> 753.  Not for the walk's propose, forward and accept kernels: a short run that
// captures and replays 61 of them per stage took 5.4 ms instead of 4.6.
// One kernel reads before its wait: mlp_layer_tc_kernel its packed weights.  What writes them has to end two
// launches back or more, with a kernel in between that waits (split_rows_kernel, in ag_mlp_forward_tc).
template <class... P, class... A>
inline void launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<A&&>(args)...);   // launch_status() reports its error
}
// checks a kernel launch and returns the ABI status
inline int launch_status(const char* name) { return cuda_status(cudaGetLastError(), name); }

}  // namespace ag

#define AG_REQUIRE(cond, ...)                                   \
    do {                                                        \
        if (!(cond)) return ::ag::set_error(AG_ERR_ARG, __VA_ARGS__); \
    } while (0)
