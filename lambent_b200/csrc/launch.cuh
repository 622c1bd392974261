// launch.cuh - programmatic dependent launch of kernels that follow one another in a stream.
//
// A kernel launched with launch_next may be set up, and its blocks started, as the previous kernel's last
// blocks exit; its wait_previous() holds it until that kernel's results are complete and visible.  Every
// kernel launched so calls it before it touches memory that another kernel writes or reads.  Without the
// launch attribute, and after a kernel that was launched otherwise, it does nothing.  Such memory is read by
// plain loads: the read-only path (__ldg, const __restrict__ parameters) is for what no kernel writes while
// this one exists, and it exists while the previous one still writes.
//
// It trims the 2-3 us between dependent kernels: 128x128, 1 spp, 5 bounces 158 -> 133 us; 256x256, 16 spp, 8
// bounces 1,417 -> 1,366.  Letting the next kernel start earlier, when all blocks of the previous one have
// (griddepcontrol.launch_dependents at their beginning), made every larger render slower (1,434 us; 1080p
// icosphere field 78.2 -> 79.2 ms): blocks that start while another kernel holds an SM keep that kernel's
// split of shared memory and L1.
#pragma once
#include <cuda_runtime.h>

#include "host_steps.h"

namespace lam {

__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... T>
inline cudaError_t launch_next(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const T&... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &attr;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

// Dependent launches of one call on a stream, each of which reads what those before it wrote.
struct Launches {
    cudaStream_t st;
    Steps<cudaError_t> steps;
    explicit Launches(cudaStream_t stream) : st(stream) {}
    template <class... P, class... T>
    void next(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, const T&... args) {
        steps([&] { return launch_next(kernel, grid, block, smem, st, args...); });
    }
    // The first failure, which is then no longer the runtime's last error either.
    cudaError_t status() const {
        if (steps.status != cudaSuccess) (void)cudaGetLastError();
        return steps.status;
    }
};

}  // namespace lam
