// Programmatic dependent launch, used by the kernels of an SpMV.
//
// The calls of a solver follow one another on a stream, and a kernel of a few microseconds loses as much again in the gap before
// the next one. A kernel launched by launch_pdl() may start while the one before it drains. Until grid_wait() has returned
// (everything earlier on the stream has then finished and its writes are visible) it touches only what no kernel writes: the
// plan's arrays. What other kernels write (x) is read after the wait, by ordinary loads in program order: `ld.global.nc` would
// promise that nobody writes x while the kernel exists. What the code relies on: every thread that stores anything waits first, and in
// every CTA some thread does, so that a kernel finishes only after everything before it on the stream has; waiting for the one
// kernel before is then waiting for all.
//
// grid_release() lets the next kernel start when all CTAs of this one have called it (or ended). Most kernels call it after their
// wait, so that one kernel at most is waiting behind the running one. k_clear, k_tiled, k_tiled_units and k_rows call it before: the
// two in the middle load the head of their stream meanwhile. Several kernels may then be waiting, which costs their place on the SMs and nothing else: they
// still store nothing before everything earlier has finished, and a kernel's CTAs are all on the device before the next one's are.
#ifndef ASP_LAUNCH_H
#define ASP_LAUNCH_H

#include <cuda_runtime.h>

namespace asp
{
#ifdef __CUDACC__
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// the wait before the first use of x, in whichever loop that is
struct WaitOnce
{
    bool done = false;
    __device__ __forceinline__ void operator()()
    {
        if (done) return;
        grid_wait();
        grid_release();
        done = true;
    }
};

// x: as volatile PTX, which stays behind the wait and keeps its order
__device__ __forceinline__ float ld_x(const float *p)
{
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double ld_x(const double *p)
{
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

template <class... A>
cudaError_t launch_pdl(void (*kernel)(A...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    void *p[] = {(void *)&args...};
    return cudaLaunchKernelExC(&cfg, (const void *)kernel, p);
}
#endif
} // namespace asp
#endif
