// launch.cuh - kernels of one stream's chain launched before their predecessor ends.
//
// A small frame is a chain of some twenty launches of a few microseconds each,
// and between two of them the chip waits for the next launch to arrive and
// its blocks to start.  lux::launch starts a kernel as soon as the one before it
// in the stream runs (programmatic dependent launch); the kernel waits in its
// first statement, after_previous, for that kernel's end.  Cornell preview
// (385 rays, 22 launches) 145 -> 112 us, dense Cornell 205 -> 176; frames of
// milliseconds are the same.
#pragma once
#include <cuda_runtime.h>

namespace lux {

// The first statement of every kernel that launch() starts, reached by all its
// threads: waits for the end of the kernel before it in the stream, whose
// results are visible from here on, then lets the next kernel start (to wait in
// its turn; so at most one waiting kernel shares the chip).  What the kernel
// before it may have written is read by ordinary loads: neither by __ldg nor
// through a const __restrict__ pointer parameter.  Those promise memory that is
// constant while this kernel lives, and it lives while that kernel still
// writes, so such a load may be moved up or take a line read too early.  What
// was complete when the kernel before it began (scene data, the cell
// directories in a resolve, the corners in a children pass) may be read so.
__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// kernel<<<grid, block, smem, st>>>(args...) for a kernel that begins with
// after_previous.  After anything but a kernel it is an ordinary launch.
template <typename... P, typename... A>
inline void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
    cudaLaunchAttribute early[1];
    early[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = early;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace lux
