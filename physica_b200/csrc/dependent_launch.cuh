// Kernel launches that overlap the end of the stream's previous kernel (programmatic dependent launch).
//
// A substep is a chain of 15 to 70 short kernels.  Launched the plain way each waits until its predecessor
// has completed and then pays its own launch latency, 2 to 3 us a kernel.  Here a kernel's blocks are
// placed on the SMs once its predecessor's last blocks have exited, and wait there for its completion and
// its writes.  Plain against this, ms: 5k-particle step 0.231 -> 0.192, 103k with boundary 0.619 -> 0.559,
// 64k gradient step 1.040 -> 0.967, 270k DFSPH step 1.165 -> 1.102, 131k PCISPH gradient step 1.688 ->
// 1.609, 1M WCSPH step 0.638 -> 0.618; 1M step (long kernels) 3.48 both ways.
//
// No kernel lets its successor start earlier still (cudaTriggerProgrammaticLaunchCompletion): the waiting
// blocks then hold registers and shared memory through the predecessor's last wave.  With it the same
// steps took 0.196, 0.713, 1.078, 1.159, 1.633, 1.037 and 3.56 ms.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace pbf {

// The first statement of every kernel launched by launch_after(), in every thread, before any memory access:
// waits until the stream's previous kernel has completed and its writes are visible.  As that one waited
// for its own predecessor, a kernel sees all that the stream ran before it.  Returns at once in a kernel
// whose predecessor is not a kernel.
__device__ __forceinline__ void after_predecessor() {
    cudaGridDependencySynchronize();
}

template <class T>
struct SameType {
    using type = T;   // keeps a parameter out of the deduction: arguments convert as in a call
};

template <class... Parameters>
inline void launch_after(cudaStream_t stream, void (*kernel)(Parameters...), const unsigned blocks, const unsigned threads,
                         typename SameType<Parameters>::type... arguments) {
    cudaLaunchAttribute overlap{};
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(blocks);
    config.blockDim = dim3(threads);
    config.stream = stream;
    config.attrs = &overlap;
    config.numAttrs = 1;
    cudaLaunchKernelEx(&config, kernel, arguments...);   // errors: cudaGetLastError()
}

// Multiprocessors of the current device (0 after an error).
inline uint32_t multiprocessors() {
    int device = 0, count = 0;
    if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
        return 0u;
    return static_cast<uint32_t>(count);
}

// Threads of `kernel` that are resident at once on the current device, in blocks of `block`.
template <class... Parameters>
inline cudaError_t one_wave(void (*kernel)(Parameters...), const int block, uint32_t& threads) {
    int blocks = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, block, 0);
    threads = multiprocessors() * static_cast<uint32_t>(blocks) * static_cast<uint32_t>(block);
    return e;
}

}  // namespace pbf
