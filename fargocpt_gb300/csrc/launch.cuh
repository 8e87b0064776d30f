// Launches that overlap the start of a kernel with the end of the one before it
// in the stream (programmatic dependent launch): the kernel is put on the
// device once every block of its predecessor has started, and its blocks wait
// in follow_predecessor() until the predecessor has completed and its writes are
// visible.  What is hidden is the launch itself, about 2 us, which a small disk
// pays for each of its ten kernels and the disk force's two.  Every kernel launched this way must
// call follow_predecessor() before anything else, so that completion stays
// transitive along the stream.
#pragma once

#include <cuda_runtime.h>

namespace fgpu {

__device__ __forceinline__ void follow_predecessor()
{
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class T>
struct as_is {
    using type = T;
};

template <class... P>
inline void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                   typename as_is<P>::type... args)
{
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
    cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace fgpu
