// Shared helpers of the dm_gb300 CUDA library (sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "dm_gb300.h"

namespace dmg {

// Kernels launched by this library since load (dm_kernel_launch_count()).
void count_launch(int k = 1);

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

inline int64_t pow4(int e) { return int64_t(1) << (2 * e); }

// Stride (in coefficients) of qubit q's Pauli axis in an n-qubit state.
inline int64_t axis_stride(int n, int q) { return pow4(n - 1 - q); }

inline size_t dtype_size(int dtype) { return dtype == DM_F64 ? 8 : 4; }

inline bool valid_dtype(int dtype) { return dtype == DM_F64 || dtype == DM_F32; }

inline bool valid_n(int n) { return n >= 1 && n <= DM_MAX_QUBITS; }

// Number of SMs of the current device (cached per device).
int sm_count();

// Raise func's dynamic shared-memory limit to `bytes` on the current device
// (once per kernel and device; the attribute is per device).
cudaError_t ensure_max_dynamic_smem(const void *func, int bytes);

// Check the launch that was just enqueued.
inline int launch_status() {
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? DM_OK : DM_ERR_CUDA;
}

// Launch whose blocks may start while the stream's previous kernel still runs: they set up (barriers,
// TMEM, shared memory) and then wait in grid_wait() until everything before them in the stream is
// complete and visible.  Such a kernel calls grid_wait() in every thread before it touches global
// memory, and after its TMEM is allocated.  A kernel of a few microseconds costs as much again in launch,
// set-up and tail: a training step of 12 launches took 192 us without, 165 us with; a prediction of 61
// launches 654 and 528 us; the 16 passes of 20 layers on 10 qubits 356 us, and 244 us with this, a tile
// per SM and one composition launch for all of them.
template <typename... P, typename... A>
int launch_early_if(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = early ? 1 : 0;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = 1;
    (void)cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
    count_launch();
    return launch_status();
}

template <typename... P, typename... A>
int launch_early(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...args) {
    return launch_early_if(true, kernel, grid, block, smem, s, std::forward<A>(args)...);
}

#ifdef __CUDACC__
// Wait for the kernels before this one; then let the next one's blocks start their set-up.  The second
// after the first, always: a kernel that has started knows that all before its predecessor is complete.
__device__ __forceinline__ void grid_wait() {
    asm volatile("griddepcontrol.wait;\ngriddepcontrol.launch_dependents;" ::: "memory");
}

// A pointer whose loads cannot be moved above grid_wait(): the compiler takes memory behind a const
// restrict parameter for constant over the whole kernel.
template <typename T>
__device__ __forceinline__ T *waited(T *p) {
    asm volatile("" : "+l"(p)::"memory");
    return p;
}
#endif

// Grid size for a grid-stride loop over `work` items with `threads` per block.
inline int grid_for(int64_t work, int threads, int blocks_per_sm = 8) {
    int64_t want = (work + threads - 1) / threads;
    int64_t cap = int64_t(sm_count()) * blocks_per_sm;
    if (want > cap) want = cap;
    if (want < 1) want = 1;
    return int(want);
}

}  // namespace dmg

#define DM_CHECK_ARG(cond)              \
    do {                                \
        if (!(cond)) return DM_ERR_ARG; \
    } while (0)

#define DM_CUDA_TRY(call)                                  \
    do {                                                   \
        if ((call) != cudaSuccess) {                       \
            (void)cudaGetLastError();                      \
            return DM_ERR_CUDA;                            \
        }                                                  \
    } while (0)
