// asv_follow.cuh -- kernels that start while the one before them ends.
//
// A Lloyd iteration is a chain of some ten kernels, the flow of fifty, and
// between two of them the GPU drained and filled again.  A kernel launched by
// asv_launch_follow may start when all blocks of the one before on its stream have
// called asv_follow (or ended, with asv_follow_wait); its own call, before it
// touches global memory, waits until that kernel has ended and its writes are
// visible.  Each block calls it, also one without work: the next kernel relies on
// this one's end to know that those before have ended.  It lets the next kernel
// start only after its own wait, so at most two kernels of a chain are on the GPU
// at once.  What the kernel before writes is not read-only while this one runs:
// it is read by plain or L2 loads behind asv_follow, through pointers that are not
// const __restrict__ (__ldg, or a load that the compiler makes one, may be moved
// ahead of the wait).
// The passes of the flood let the next kernel start at their end only: blocks that
// start beside the last ones of a pass crowd on the SMs that are free first, which
// then have more tiles (1280x720x30, ten iterations: 20.0 ms so, 19.33 with the
// wait alone).  Launched plainly, 19.39 ms; the 320x240x85 clip 8.69, so 8.58, the
// 240x160x30 one with its full ladder 3.39, so 3.30; the flow of 640x480x16 3.60,
// so 3.49.
#pragma once

#include <cuda_runtime.h>

#ifdef __CUDACC__

__device__ __forceinline__ void asv_follow()
{
    asm volatile("griddepcontrol.wait;\ngriddepcontrol.launch_dependents;\n" ::: "memory");
}

// without letting the next kernel start before this one's end
__device__ __forceinline__ void asv_follow_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// A load of what the launch before wrote: as a volatile statement it stays behind
// the wait, as asm statements keep their order, but may move across other memory
// accesses, where a plain load holds its registers (k_fl_iter's flow, 640x480x16:
// plain 3.02 ms, so 2.96; the list form's labels, 640x480x40 with 12000 seeds, eight
// iterations: 18.76, so 18.50)
__device__ __forceinline__ float asv_load_behind(const float *p)
{
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ int asv_load_behind(const int *p)
{
    int v;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// follow: the operation before on st is a kernel that calls asv_follow (or one
// that doesn't: then this one starts after its end); false: a plain launch, for
// kernels behind a memset, a copy or an event of another stream
template <typename... P, typename... A>
inline void asv_launch_follow(bool follow, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                              A... args)
{
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = follow ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

#endif
