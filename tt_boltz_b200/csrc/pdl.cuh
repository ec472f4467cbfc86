// Programmatic dependent launch.
//
// A kernel launched with launch_pdl may start while its predecessor on the stream drains: what stands before
// grid_dependency_wait() (barriers, tensor memory, descriptors) overlaps the predecessor's tail and the launch itself.
// Nothing that the predecessor wrote, or reads, may be touched before the wait, and weights count as written: a program may
// have updated them on the stream.  Every CTA executes the wait, on every path, so that a kernel's completion implies that of
// all before it.  Kernels launched this way read global memory with plain loads: an ld.global.nc (__ldg, const __restrict__)
// may be moved above the wait.
#pragma once

#include <atomic>
#include <utility>

#include "common.cuh"

namespace b200pf {

__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... KArgs, class... Args>
static inline int launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    B200PF_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...));
    count_launch();
    return B200PF_OK;
}

// Multiprocessors of the current device, asked for once per device.
static inline int device_multiprocessors(int* out) {
    static int known[64] = {0};
    int dev = 0;
    B200PF_CUDA(cudaGetDevice(&dev));
    int sms = dev >= 0 && dev < 64 ? known[dev] : 0;
    if (sms == 0) {
        B200PF_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        if (dev >= 0 && dev < 64) known[dev] = sms;
    }
    *out = sms;
    return B200PF_OK;
}

// The same on CTA pairs (clusters of two), for kernels that don't name their cluster's size themselves.
template <class... KArgs, class... Args>
static inline int launch_pdl_pairs(void (*kern)(KArgs...), unsigned pairs, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    B200PF_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...));
    count_launch();
    return B200PF_OK;
}

// How many CTA pairs of a kernel are resident at once on the current device (not every SM can be half of a pair): the grid of a
// persistent pair kernel.  Asked for once per kernel and device.
template <auto KERN>
static inline int resident_pairs(int threads, int smem, int* out) {
    static std::atomic<int> known[64];
    int dev = 0, sms = 0, rc;
    B200PF_CUDA(cudaGetDevice(&dev));
    int n = dev >= 0 && dev < 64 ? known[dev].load(std::memory_order_relaxed) : 0;
    if (n == 0) {
        if ((rc = device_multiprocessors(&sms)) != B200PF_OK) return rc;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(sms / 2 * 2));
        cfg.blockDim = dim3((unsigned)threads);
        cfg.dynamicSmemBytes = (size_t)smem;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 2;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        B200PF_CUDA(cudaOccupancyMaxActiveClusters(&n, KERN, &cfg));
        B200PF_REQUIRE(n > 0, B200PF_ERR_CUDA, "no CTA pair fits on this device");
        if (dev >= 0 && dev < 64) known[dev].store(n, std::memory_order_relaxed);
    }
    *out = n;
    return B200PF_OK;
}

// The multiprocessors that a launch sizes its grid for: the device's, or fewer while this thread holds a CtaLimit.
inline thread_local int cta_limit = 0;
struct CtaLimit {
    const int before;
    explicit CtaLimit(int n) : before(cta_limit) { cta_limit = n; }
    ~CtaLimit() { cta_limit = before; }
    CtaLimit(const CtaLimit&) = delete;
    CtaLimit& operator=(const CtaLimit&) = delete;
};
static inline int multiprocessors(int* out) {
    const int rc = device_multiprocessors(out);
    if (rc == B200PF_OK && cta_limit > 0 && cta_limit < *out) *out = cta_limit;
    return rc;
}

}  // namespace b200pf
