// pdl.cuh — programmatic dependent launch for the solvers' iteration kernels.
//
// A kernel launched with programmatic stream serialisation may start while its predecessor in
// the stream is still draining; it waits in pdl_wait() (griddepcontrol.wait) before reading
// anything the predecessor wrote, which overlaps the launch and block ramp-up of consecutive
// iteration kernels.  For a plain launch pdl_wait() is a no-op.
//
// A grid of at most one block an SM also lets its successor start as soon as it has waited itself
// (griddepcontrol.launch_dependents), instead of when its blocks have exited: a 64x32x32 mixed
// step 3.31 -> 3.20 ms.  Larger grids need the SMs' slots for their own blocks: with the early start
// for up to 300 blocks the 256x128x128 step went from 13.80 to 14.17 ms, for all grids 14.41.
#pragma once
#include <cuda_runtime.h>

namespace suli {

constexpr unsigned int kPdlEarlyBlocks = 148;   // one an SM of a B200, the only part this is built for
__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (gridDim.x * gridDim.y * gridDim.z <= kPdlEarlyBlocks) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// launch with programmatic stream serialisation (the kernel calls pdl_wait before its loads)
template <typename... KArgs, typename... Args>
static void pdl_launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace suli
