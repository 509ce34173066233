// Launches that start before the launch in front of them has ended (programmatic dependent launch): the small kernels that bound
// and re-lay the dense operand let the next one start as soon as their own last CTA has, so that its launch and its set-up
// (barriers, tensor memory) run beside them instead of after them.  A kernel launched this way calls wait_for_previous_launch()
// before it touches what another launch writes or still reads, and in any case before it ends: what waits for it has then waited for all
// before it.  column_range_kernel (qcsr_transpose_digits.cu) reads G and writes its parts first: the launch in front of it is the first of its call,
// which touches neither and was not made early itself.
// 5,000 x 2,000 at N = 64, decoded tiles: 31.3 -> 24.0 us a call; 20,000 x 4,096 Blocked-ELL 33.1 -> 28.9.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace cb200 {

// until the launches in front have ended and their writes are visible; returns at once in a launch that was not made early
__device__ __forceinline__ void wait_for_previous_launch() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// the next launch of the stream may start once every CTA of this one has come here
__device__ __forceinline__ void let_next_launch_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// `early`: the launch in front on the stream is a kernel of the same call
template<typename... P, typename... A>
cudaError_t launch_kernel(bool early, void (*kernel)(P...), dim3 grid, unsigned threads, std::size_t smem, cudaStream_t stream, A... args) {
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &attribute;
    config.numAttrs = early ? 1u : 0u;
    return cudaLaunchKernelEx(&config, kernel, static_cast<P>(args)...);
}

} // namespace cb200
