// Launching a kernel so that its start overlaps the end of the one before it.
#pragma once

#include "common.cuh"

namespace mask {

// Programmatic dependent launch: a kernel of this library starts while the kernel before it in the stream is still
// draining (once all of that kernel's blocks have begun, if it is one of ours, or ended), sets itself up and then
// waits for it to finish.  Nothing but the plan's own tables, which are complete when mask_plan_create returns, is
// read before the wait.  Between the product and its fix-up pass, or from one product to the next, this hides
// a launch: 3 of 14 us for a product of 1000 rows.
__device__ __forceinline__ void wait_for_previous_kernel() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_kernel_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... Params, typename... Args>
int launch_overlapped(void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    MASK_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...));
    return MASK_OK;
}

}  // namespace mask
