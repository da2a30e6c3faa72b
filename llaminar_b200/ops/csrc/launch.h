// Host-side launch helper: programmatic dependent launch (PDL).
//
// A kernel launched through `launch_pdl` may be scheduled while its predecessor in the stream is still running: as soon
// as every CTA of the predecessor has executed `griddepcontrol.launch_dependents` (or exited), the CTAs of this kernel
// start, run their prologue (shared-memory carve-up, barrier init, TMEM allocation) and block in `griddepcontrol.wait`
// until the predecessor has finished and its writes are visible.  That hides the launch gap and the prologue of the
// many small kernels of a decode step, inside CUDA graphs as well.  Kernels launched this way call `pdl_trigger()` first
// and `pdl_wait()` before they touch global memory (common.cuh).  A predecessor that never triggers (any other kernel)
// simply keeps the ordinary stream order.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace llm {

// SMs of the current device.  CTAs of the persistent kernels wait for one another, so a launch has no more of them than fit at once.
inline int sm_count() {
    static int n = 0;
    if (!n) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev); }
    return n > 0 ? n : 148;
}

// CTAs of two matrices that share a launch of `ctas` in all: by bytes, no more than `most` of either and at least one.
// {0, 0}: there is no room for two.
struct Shares { int first, second; };
inline Shares share_ctas(double bytes_a, double bytes_b, int most_a, int most_b, int ctas) {
    if (ctas < 2) return {0, 0};
    int b = (int)(ctas * bytes_b / (bytes_a + bytes_b) + 0.5);
    if (b > most_b) b = most_b;
    if (b > ctas - 1) b = ctas - 1;
    if (b < 1) b = 1;
    int a = ctas - b;
    if (a > most_a) a = most_a;
    if (a < 1) a = 1;
    return {a, b};
}

inline bool& pdl_enabled() {
    static bool on = true;
    return on;
}

template <class... KArgs, class... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(std::forward<Args>(args))...);
}

}  // namespace llm
