// Launches of kernels each of which starts while the one before it drains, and
// the scalars of a step, handled inside the fused kernels.
//
// A step of a small grid is two kernels of a few microseconds; the gap between
// two of them is mostly the next one's launch. Launched with programmatic stream
// serialization, a kernel's blocks are set up as soon as every block of the
// one before has called grid_go() or ended; its first statement, grid_wait(),
// waits until that one is complete and its writes are visible. Every kernel
// launched this way waits first, so each sees everything before it, as in
// plain stream order. Measured, with the scalars' own launches folded in:
// 333^2 cells in binary32, 40 steps in graphs 1.35 -> 1.26 ms; 128 boxes in 3-D,
// 30 steps 36.3 -> 34.7 ms. (Large 2-D grids lose by the folding: tj_mixed.cu.)
#pragma once

#include <cuda_runtime.h>

#include "tj_types.h"

namespace tj {

__device__ __forceinline__ void grid_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void grid_go()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Whether this is thread 0 of the last block of the grid to get here; called
// by every thread at the end of a kernel. What every block wrote before is
// visible to it. The scalars of a step are then handled by the kernel that
// ends a stage instead of by a launch of one thread.
__device__ __forceinline__ bool last_block(DevScalars* s)
{
    __syncthreads();
    if (threadIdx.x != 0) return false;
    __threadfence();
    if (atomicAdd(&s->ticket, 1u) != gridDim.x * gridDim.y - 1) return false;
    s->ticket = 0;
    __threadfence();
    return true;
}

// A step's dt from the CFL minimum (main.cpp:128-143): dt, and whether the run
// is over (t has reached t_end).
__device__ __forceinline__ bool step_dt(const DevScalars* s, double cfl, double raw, double& dt)
{
    if (!(s->t < s->t_end)) return true;
    dt = __dmul_rn(cfl, raw);  // not contracted, in whatever unit this is compiled
    if (__dadd_rn(s->t, dt) > s->t_end) dt = __dsub_rn(s->t_end, s->t);
    if (s->n < 5) dt = __dmul_rn(dt, 0.2);
    return false;
}

// Takes the CFL minimum and re-arms it; with clamp, sets the step's dt.
__device__ __forceinline__ void finalize_dt(DevScalars* s, double cfl, int clamp)
{
    const double raw = __longlong_as_double((long long)*(volatile unsigned long long*)&s->dtmin_bits);
    s->dtmin_raw = raw;
    s->dtmin_bits = 0x7FEFFFFFFFFFFFFFull;
    if (!clamp || s->done) return;
    double dt;
    if (step_dt(s, cfl, raw, dt)) s->done = 1;
    else s->dt = dt;
}

// The end of a step (main.cpp:121 t += dt; the NaN stop of 183-187).
__device__ __forceinline__ void end_step(DevScalars* s)
{
    if (*(volatile int*)&s->nan_flag) {
        s->done = 1;
        atomicCAS(&s->status, 0, TJ_ERR_NAN);
        return;
    }
    s->t = __dadd_rn(s->t, s->dt);
    s->n += 1;
}

// kernel<<<grid, threads, smem, st>>>(args...), overlapping its launch with the
// kernel before it on the stream. The kernel must begin with grid_wait().
// overlap = false: a plain launch (events recorded around single kernels).
template <class... Params, class... Args>
inline void launch(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t st, bool overlap,
                   const Args&... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

}  // namespace tj
