// Shared by every .cu in the shim: status plumbing and launch helpers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/clpeak_b200_kernels.h"

namespace clpk {

// Record a detail string for clpk_last_error() (thread-local).
void set_error(const char *fmt, ...);

// Maps a CUDA error to CLPK_ERR_CUDA / CLPK_ERR_NO_DEVICE and records the detail.
int cuda_fail(cudaError_t e, const char *what);

// The current device must be compute capability 10.x; anything else is refused
// (there is no fallback path).
int require_sm100();

int num_sms();          // of the current device (cached per device)
int smem_optin_bytes(); // of the current device

// Value of a CLPK_TUNE_* knob, or -1 when neither the environment (read once) nor
// clpk_set_tuning has set it.
int tuning(int knob);

// fp32 (CUDA cores) and fp64 (DMMA) GEMMs, simt_gemm.cu; dtype is CLPK_DT_F32 or CLPK_DT_F64; *status is cleared.
int launch_simt_gemm(int dtype, const void *a, const void *b, void *c, uint32_t m, uint32_t n, uint32_t k, float alpha,
                     uint32_t *status, cudaStream_t s);

// what those two types ask of their operands
int check_simt_gemm(int dtype, const void *a, const void *b, const void *c, uint32_t m, uint32_t n, uint32_t k);

// microseconds that its plan for an fp32 product is estimated at
float simt_f32_estimate(uint32_t m, uint32_t n, uint32_t k);

// clpk_gemm_plan of those two types
void simt_gemm_plan(bool f64, uint32_t m, uint32_t n, uint32_t k, uint32_t *tile_n, uint32_t *splits, uint32_t *wide);

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

} // namespace clpk

namespace clpk {

// Launches a kernel with the programmatic-serialisation attribute: its first CTAs take their places under the tail of
// the kernel before it in the stream.  The kernel must therefore wait (griddep_wait) before it touches memory.
template <typename... Params, typename... Args>
int launch_behind(void (*kernel)(Params...), const char *what, unsigned grid, int threads, size_t smem, cudaStream_t s, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
    return e == cudaSuccess ? CLPK_OK : cuda_fail(e, what);
}

} // namespace clpk

#define CLPK_CUDA(call)                                          \
    do {                                                         \
        cudaError_t e__ = (call);                                \
        if (e__ != cudaSuccess)                                  \
            return ::clpk::cuda_fail(e__, #call);                \
    } while (0)

#define CLPK_REQUIRE(cond, ...)                                  \
    do {                                                         \
        if (!(cond)) {                                           \
            ::clpk::set_error(__VA_ARGS__);                      \
            return CLPK_ERR_BAD_ARG;                             \
        }                                                        \
    } while (0)

#define CLPK_LAUNCH_CHECK(name)                                  \
    do {                                                         \
        cudaError_t e__ = cudaGetLastError();                    \
        if (e__ != cudaSuccess)                                  \
            return ::clpk::cuda_fail(e__, "launch " name);       \
    } while (0)
