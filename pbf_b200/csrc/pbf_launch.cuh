// Programmatic dependent launch: a kernel launched with it may start before the
// kernel before it in the stream (or captured graph) is complete, and waits at
// pdl_wait until it is and its writes are visible. A kernel of such a chain calls
// pdl_wait in every thread before it touches memory or returns, so that its own
// completion implies that of everything before it.
#pragma once
#include <cuda_runtime.h>

namespace pbf {

// Lets the next kernel of the chain launch once every block has called this. The
// substep's kernels do not: waiting blocks of the next kernels then take room from
// the running one (a frame of 32,768 particles: 189 us without it, 199 with the call
// before the epilogues and 237 at the top; without programmatic launches 193).
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// True when this launch is to be refused (pbf_debug_fail_launch; pbf_capi.cu).
bool refuse_launch();

// Launches k, with programmatic stream serialisation when pdl is set; 0 on success. (A
// refused launch is also the runtime's last error, which the substep's capture checks.)
template <typename... P, typename... A>
int launch(bool pdl, void (*k)(P...), int grid, int block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(refuse_launch() ? 0u : (unsigned)grid);  // (the runtime refuses an empty grid)
    c.blockDim = dim3((unsigned)block);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&c, k, P(args)...) == cudaSuccess ? 0 : -1;
}

}  // namespace pbf
