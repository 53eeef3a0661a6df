// Kernel launches that may begin before the kernel ahead of them in the stream has ended (programmatic dependent launch).
//
// Every kernel of a training step (not those of comm.cu, which exchange gradients) sets itself up (barriers, tensor memory, shared
// memory), then calls dependent_begin() before it touches global memory: that waits until the kernels ahead are complete and their
// writes visible, and lets the next kernel of the stream be set up in turn. As a kernel lets the next one in only after its own wait, at most two kernels of a stream are on the chip, and
// a kernel that is not launched this way (another library's, a copy, an exchange kernel) is ordered as ever.
// What it saves is the gap between two launches, 1 to 2 us, and the set-up, 1 to 3 us. What it costs: the CTAs of the next kernel take
// shared memory from the L1 of a kernel that still runs, find little of it themselves beside one that asked for all shared memory, and
// take SMs from the other stream. See OverlapLaunches and OverlapFp32Launches in engine.cu for where it pays.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace mgt {

__device__ __forceinline__ void dependent_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// For a pointer whose first read follows dependent_begin() without a branch or barrier between them: a read through the read-only
// path depends on nothing else that the compiler sees.
template <class T>
__device__ __forceinline__ T* after_begin(T* p) {
    asm volatile("" : "+l"(p));
    return p;
}

// Where a kernel goes, and whether it may begin before the one ahead of it has ended.
struct LaunchOn {
    cudaStream_t stream;
    bool overlap;
    LaunchOn(cudaStream_t s, bool o) : stream(s), overlap(o) {}
    operator cudaStream_t() const { return stream; }
};

template <class... Params, class... Args>
inline cudaError_t Launch(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, LaunchOn on, Args&&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = on.stream;
    config.attrs = &attr;
    config.numAttrs = on.overlap ? 1 : 0;
    return cudaLaunchKernelEx(&config, kernel, std::forward<Args>(args)...);
}

}  // namespace mgt
