// Programmatic dependent launch: a kernel launched with launch_pdl() may be scheduled while the
// kernel before it on the stream is still running. Its CTAs take the SMs the predecessor's CTAs
// leave, run their set-up (barrier initialisation, tensor-memory allocation, descriptor
// prefetch) and then block in pdl_wait() until the predecessor has completed and its writes
// are visible. That hides the launch latency and the ramp of each of the 20-odd kernels of a
// network behind the tail of the previous one. A kernel launched this way reads and writes no
// global memory before pdl_wait(), with one exception: operands that no kernel in flight writes, as
// the launch was told (ConvArgs::params_early). And it releases its successor only behind its own
// pdl_wait(): so when a kernel starts, all but the one in front of it have completed, and what
// that one writes is what its launch recorded (last_launch_writes). A kernel launched without the
// attribute executes the two instructions as no-ops, and one that never releases is complete when
// its successor starts.
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "tuning.h"

namespace mb200 {

#if defined(__CUDACC__)
// Releases the NEXT kernel for scheduling (it still waits for this one to complete before it
// touches memory); only behind a pdl_wait().
__device__ __forceinline__ void pdl_release() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void pdl_start() {
    pdl_wait();
    pdl_release();
}
#endif

// the memory that a launch writes
struct Writes {
    const void* first;
    size_t bytes;
};

// What the library's last launch on a stream writes, kept per stream (abi.cu). Held for the launch,
// so that records come in the order of the launches.
class LaunchRecord {
public:
    LaunchRecord(cudaStream_t st, const Writes& writes);
    ~LaunchRecord();
    // (a launch that failed leaves the one before it the last, of which nothing is known any more)
    cudaError_t result(cudaError_t e) {
        if (e != cudaSuccess)
            forget();
        return e;
    }

private:
    void forget();
    void* slot_;
};
// May the last launch on the stream write any of these bytes? (true where it is not known)
bool last_launch_writes(cudaStream_t st, const void* p, size_t bytes);

template <class... KArgs, class... Args>
inline cudaError_t launch_pdl(
        const Writes& writes, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
        Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tuning().pdl ? 1 : 0;
    LaunchRecord record(st, writes);
    return record.result(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...));
}

// The same with `cluster` consecutive CTAs of the grid as one thread-block cluster (1: none).
template <class... KArgs, class... Args>
inline cudaError_t launch_pdl_cluster(
        const Writes& writes, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, int cluster, cudaStream_t st,
        Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (cluster > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)cluster;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    if (tuning().pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    LaunchRecord record(st, writes);
    return record.result(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...));
}

}  // namespace mb200
