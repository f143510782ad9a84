// Launches of kernels that follow one another in a stream: a chained kernel may be set up while its predecessor
// still runs, and its blocks wait at chain_begin() until that one is complete and its writes are visible
// (programmatic dependent launch).  Chains of short kernels are otherwise bound by the gaps between them (mesh sum of 99 998 charges in nine
// kernels 148 -> 136 us, learned correction of 64 000 ions in seven 90 -> 70 us).  Not for a kernel whose few long blocks
// have to spread over the chip (launch_gather_t in mesh_kernels.cuh).
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace pdb {

// First statement of every chained kernel, before any access to memory: lets the next kernel of the stream be set
// up, then waits for the previous one.  Every kernel of a chain waits here, so "the previous one is complete"
// holds for all before it.  Without the launch attribute both instructions do nothing.
__device__ __forceinline__ void chain_begin() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// kernel<<<grid, block, shm, s>>>(args...), chained; failures are picked up by PD_LAUNCHED().  Not inside a stream
// capture: in a captured step two branches share the SMs, and blocks of the one that wait for their turn hold
// registers and shared memory that the other's could use (10 steps of 64 000 ions 1036 -> 1111 us, of 12 batched
// melts 814 -> 964 us with chained graph edges).
template <typename... P, typename... A>
inline void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t shm, cudaStream_t s, A &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = shm;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(s, &capturing);
    cfg.numAttrs = capturing == cudaStreamCaptureStatusNone ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace pdb
