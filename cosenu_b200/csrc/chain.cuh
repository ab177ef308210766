// Launches that overlap the end of the previous one: programmatic dependent
// launch.
//
// A stage of a small grid, or one GEMM of a training step, runs for a few
// microseconds, of which one to two are the gap between two launches and the
// prologue (barriers, tensor memory, tensor maps, tables).  A chained launch's
// blocks start in free slots once every block of the launch before it has
// started, do the prologue and wait there.
//
// The previous launch says when (next_launch): the stage kernels after a block's
// last chunk, the training kernels ahead of the epilogue.  Said at a kernel's
// start, several launches' waiting blocks pile up in the free slots, and a stage
// on fewer blocks than slots ends up two to an SM beside idle ones.  us per pass,
// plain / at the start / after the last chunk: 100 steps of 1024 x 64 FV cells
// 3094 / 3456 / 2812; one step of 600 x 32 26.6 / 32.1 / 24.6; 50 steps of
// 2400 x 32 with analysis 2363 / 2570 / 2213; 50 FD steps of 1000 x 37 966 / 872 /
// 862; 16 ensemble members 8540 / 8636 / 8413; grids of a millisecond a step
// the same.  Training, 2000 rows in batches of 64: 2880 / 2410 / 2290.
//
// Rules: every thread of a chained kernel calls previous_launch() before its
// first access to memory that an earlier launch reads or writes; before it, only
// what no kernel of the chain writes.  It returns once the previous launch has
// ended with its memory visible, and that launch in turn had waited for its own
// predecessor, so the order between launches is the stream's.  `after` is set
// only where the previous operation on the stream is a launch of the same call.
#pragma once

#include <cuda_runtime.h>

// Lets the next launch's blocks start where there is room.
__device__ __forceinline__ void next_launch()
{
    asm volatile("griddepcontrol.launch_dependents;");
}

// Waits for the previous launch (returns at once in an ordinary launch).
__device__ __forceinline__ void previous_launch()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... P, class... A>
inline cudaError_t launch_after(bool after, void (*kernel)(P...), int blocks, int threads, int smem,
                                cudaStream_t s, A &&...args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)blocks);
    c.blockDim = dim3((unsigned)threads);
    c.dynamicSmemBytes = (size_t)smem;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = after ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, static_cast<A &&>(args)...);
}
