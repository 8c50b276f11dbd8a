// ccc_runtime.cuh — launch accounting shared by the library's translation units.
//
// Every kernel launch goes through CCC_LAUNCH, which counts it and, while per-kernel
// timing is on (ccc_timing_begin / ccc_timing_end) and the stream is not being captured
// into a graph, brackets it with CUDA events on the launching stream.  Definitions live in
// ccc_capi.cu.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace ccc {

// launches since load (exact when one host thread launches at a time)
extern std::atomic<int64_t> g_launches;
// elementary functions of the continuous-collision solver (MathLib)
extern int g_math_lib;

void timing_before(const char* name, cudaStream_t s, int* slot);
void timing_after(int slot, cudaStream_t s);
// per-kernel timing is on: work that would overlap on a second stream runs in order
bool timing_active();
int num_sms();

inline int64_t align_up(int64_t x, int64_t a) { return (x + a - 1) / a * a; }
inline int grid_for(int64_t n, int threads) { return (int)((n + threads - 1) / threads); }

// Launch of a kernel that begins with chain_begin(): it may start while the kernel before it in
// the stream drains (programmatic stream serialization).  Kernels that do not begin so must not
// be launched with it.
template <class... P, class... A>
cudaError_t launch_chain(int grid, int block, size_t smem, cudaStream_t s, void (*kernel)(P...), A&&... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace ccc

#define CCC_LAUNCH(name, s, ...)                  \
    do {                                          \
        int slot__;                               \
        ::ccc::timing_before(name, s, &slot__);   \
        __VA_ARGS__;                              \
        ::ccc::timing_after(slot__, s);           \
    } while (0)

// Run the statement(s) with LIBV bound to the current math library (MathLib) as a
// compile-time constant, for kernels templated on it.
#define CCC_WITH_LIB(...)                                              \
    do {                                                               \
        if (::ccc::g_math_lib == 0) {                                  \
            constexpr int LIBV = 0;                                    \
            __VA_ARGS__;                                               \
        } else {                                                       \
            constexpr int LIBV = 1;                                    \
            __VA_ARGS__;                                               \
        }                                                              \
    } while (0)

#define CCC_LAUNCH_CHECK()                                         \
    do {                                                           \
        cudaError_t e__ = cudaGetLastError();                      \
        if (e__ != cudaSuccess) return CCC_ERR_CUDA;               \
    } while (0)
