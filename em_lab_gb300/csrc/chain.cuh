// chain.cuh - programmatic dependent launch for the kernels of a time step.
//
// A step is a chain of short kernels on one stream (solver pass, sources, monitors), and on small grids
// the time between them (drain of the last blocks, launch, first loads) weighs: chained launches let a
// kernel's blocks start, and read what no kernel of the chain writes, while the one before still runs.
// A step without and with them: 128 x 128 x 128 cells with the far-field monitor 48 and 39 us,
// 211 x 147 x 93 with a port 68 and 57 us, 80 x 80 x 640 with the surface DFT 104 and 92 us,
// 512 x 512 x 512 with port and DFT 1298 and 1288 us.
//
// Rules that keep the chain in stream order:
//  - every chained kernel calls chain_wait() in at least one thread of the grid, and in every thread
//    before it touches what another kernel of the chain writes: the wait ends when the kernel before has
//    completed, so completion carries along the chain;
//  - solver kernels call chain_next() after their wait: when a kernel between two solver passes starts,
//    everything before the last solver pass has completed. What a monitor kernel itself wrote in the step
//    before may therefore be read ahead of the wait (past L1: __ldcg);
//  - the first launch after anything else on the stream (a copy, an event) is not chained.
// A kernel's blocks start only when every block of the kernel before has called chain_next() or left, so
// blocks that wait never keep out the ones they wait for.
//
// Only the sources start beside the solver pass. Kernels between two passes call chain_next() after
// their wait: with an earlier call the many blocks of the far-field kernels came in beside the
// solver too, and a step of the first and third sizes above took 60 and 163 us. The per-step far-field
// accumulation does not call it at all (with it the first size takes 1.5 us more; the DFT's sampling,
// which has no shared memory to speak of, gains 2.5 us from it).
#pragma once

#include <cuda_runtime.h>

namespace emlab {

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

struct Chain {
    cudaStream_t stream;
    bool chained;  // false: in full stream order, as an ordinary launch
};

template <class... P, class... A>
void launch_chained(const Chain& c, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, A&&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid, cfg.blockDim = block, cfg.dynamicSmemBytes = smem, cfg.stream = c.stream;
    cfg.attrs = &attr, cfg.numAttrs = c.chained ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace emlab
