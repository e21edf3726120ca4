// Programmatic dependent launches for chains of short kernels.
//
// A solve's step is six to ten kernels of 2-30 us on one stream, and between two of
// them the GPU stood still for about 2 us (drain, launch, first loads).  A kernel
// launched with launch_pdl() may become resident while its predecessor's last blocks
// run; its first statement is pdl_sync(), which waits until the predecessor has
// completed and its writes are visible, and then lets the next kernel of the chain
// follow in the same way.  Every thread of every block waits before it reads or writes
// memory, so a kernel still sees all earlier work of its stream, and at most two
// kernels of a chain are resident.
//
// Measured, the gaps gone and nothing else changed: serving six structures 195 -> 167
// ms, a direct solve of 893 unknowns 16.3 -> 14.0, a mixed solve of 7,844 unknowns
// 102 -> 94, an alloy bow-tie of 13,528 unknowns 555 -> 519.
//
// Blocks that arrive early go to the SMs that have room first.  A kernel of two or
// three blocks an SM can end up with most of them on a few SMs; even_smem() asks for so
// much shared memory that no SM takes more than its share.
#pragma once

#include <utility>

#include "plx_internal.h"

namespace plx {

__device__ __forceinline__ void pdl_sync() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// kern must begin with pdl_sync().
template <typename... P, typename... A>
void launch_pdl(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
    cudaLaunchAttribute at[1] = {};
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    PLX_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...));
}

inline int sm_count(int device) {
    int v = 0;
    PLX_CHECK_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device));
    return v > 0 ? v : 1;
}

// Dynamic shared memory (at least `smem`) with which `blocks` blocks spread evenly over
// `sms` SMs: only where an SM's share is below four, above which the spread hardly
// matters.  `fixed` is the kernel's static shared memory, 1 KB a block the system's.
inline size_t even_smem(int64_t blocks, int sms, size_t fixed, size_t smem) {
    const size_t share = (size_t)((blocks + sms - 1) / sms), whole = 222 * 1024;
    if (share >= 4 || share == 0) return smem;
    const size_t fits = whole / share - fixed - 1024;
    return fits > smem ? fits : smem;
}

}  // namespace plx
