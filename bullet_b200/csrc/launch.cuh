// What the kernels of a training step share: programmatic dependent launch and the step's clock.
//
// The kernels of a step follow each other on one stream.  Launched with programmatic stream serialisation, a kernel's CTAs
// may take their places while the last CTAs of the kernel before are still running; step_begin() then waits until that
// kernel has completed and its writes are visible, so nothing of a kernel that touches memory comes before it.  Every kernel
// lets its successor in as soon as its own last CTAs have places (launch_dependents).  Without the attribute both are no-ops.
// So the kernel before may still be writing when a kernel begins, and its output is read with loads that are coherent (__ldcg, plain
// ones), never through the read-only path (__ldg, ld.global.nc, const __restrict__), which wants data that nobody writes from the
// kernel's first instruction on.  What the kernels before that one wrote is finished by then.
// This takes most of the 3 us out of every boundary between two kernels of a step.
//
// Time stamps of the phases are written by the first thread of the kernels themselves: an event with timing between two
// kernels costs the stream about 2 us and the host 1.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

__device__ __forceinline__ unsigned long long clock_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// first statement of a step's kernel; `stamp`: where its start time goes, or null
__device__ __forceinline__ void step_begin(unsigned long long* stamp) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (stamp && threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0) *stamp = clock_ns();
}

// The largest magnitude of a pass, kept as the bits of |v| in one word: these order as the magnitudes do, infinity above every
// number and NaN above infinity.  A warp adds its own to the word, if there is one and it holds less.
__device__ __forceinline__ unsigned magnitude(float v) { return __float_as_uint(v) & 0x7fffffffu; }
__device__ __forceinline__ void raise_magnitude(unsigned* word, unsigned own) {
    if (!word) return;
    own = __reduce_max_sync(0xffffffffu, own);
    if ((threadIdx.x & 31) == 0 && own > __ldcg(word)) atomicMax(word, own);
}

template <class... Params, class... Args>
cudaError_t launch_step(bool chained, void (*kernel)(Params...), dim3 grid, int block, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = dim3(block);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &attr;
    config.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&config, kernel, Params(args)...);
}

}  // namespace b200
