// Kernels that start before their predecessor in the stream has finished (programmatic dependent
// launch): a kernel launched by launch_early may be resident while the previous kernel of its stream still
// runs, does what needs none of that kernel's results (tables of constants, barriers, shared-memory
// layout), and must call previous_done() before it reads or writes any memory that an earlier kernel
// touches. A kernel that calls next_may_start() lets its successor start once every CTA has called it; a
// kernel that calls neither behaves as ever. Since every early kernel waits for its predecessor's end
// before its own, the order holds along the whole stream. next_may_start() comes after previous_done(): a kernel's
// successor then starts when the kernel's predecessor has ended, and no more than two are resident. Called first,
// a third could be, whose SM may still load, for the first, the old contents of a buffer that the second writes and
// it reads itself.
//
// What an early kernel reads may be written while it is resident, so it is read with ordinary loads only:
// no __ldg, which wants memory that nothing writes for as long as the kernel runs, and no __restrict__, which
// makes such loads of plain ones and lets the compiler move them above previous_done().
//
// The passes of the slice loop call next_may_start() as their last act, so that only launch latency and
// start-up overlap: called first, successors that hold their place on an SM cost long passes 2 % and
// put two CTAs on one SM where a pass has fewer CTAs than there are SMs (exit wave of 8 x 256^2, 5 %
// slower). Measured over whole runs on one B200: exit wave of 16 x 256^2 1546 -> 1478 us, STEM 128^2
// x 256 probes 2507 -> 2430 us, HRTEM 8 x 512 x 384 1962 -> 1914 us, STEM 256^2 4403 -> 4344 us.
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "common.hpp"

namespace mtb {

__device__ __forceinline__ void previous_done() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// early = false: an ordinary launch, which starts after its predecessor's end.
template <class... P, class... A>
void launch_early(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = early ? 1 : 0;
    MTB_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
}

}  // namespace mtb
