// Launches of the wavefront's kernels, each of which follows another at once.
#pragma once
#include <cuda_runtime.h>

namespace cpppt_gb300 {

// Launches a kernel that begins with after_previous(): its CTAs take their
// places as those of the kernel before it leave, and wait there until that
// kernel's writes are visible, which hides most of the time between two
// launches (about a microsecond, and a render makes 80 to 250 of them).  Every
// CTA waits first, so the kernels still run one after the other.  SD-tree
// render, Cornell box 128x128, 64 spp, 3.59 -> 3.17 ms; training 640x360 in the
// 192k-triangle room 7.95 -> 7.73, guided 1280x720 10.05 -> 9.91; 640x360, 1
// spp on the 1M-triangle soup 1.85 -> 1.82; long kernels (1080p) unchanged.
//
// A kernel's lifetime so overlaps the writes of the one before, and a load
// through the read-only path is not ordered by the wait.  What another kernel of
// the loop writes (path state, hits, mixtures, queues, counters) is therefore
// never read through `const ... __restrict__` or __ldg, which are for what stands
// before the render: scene arrays, the guide's tree, job tables.
template <class... A, class... B>
void launch_after(void (*kernel)(A...), int grid, int threads, size_t smem, cudaStream_t st, B&&... args) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3((unsigned)threads);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute a{};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &a;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, kernel, static_cast<A>(args)...);  // a failure is the last error, as after <<<>>>
}

__device__ __forceinline__ void after_previous() { cudaGridDependencySynchronize(); }

}  // namespace cpppt_gb300
