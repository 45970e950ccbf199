// vpt_scratch.cu - stream-ordered scratch of the entry points that keep no state between calls: the ping-pong
// image of vpt_eaw_denoise_rgba, the planes of vpt_svgf_filter, the fp32 partial sums of vpt_unet_conv3x3.
//
// The device's default pool returns its memory at every synchronisation (release threshold 0), so that the next
// call maps it again: 0.5 ms of a 1920 x 1080 EAW call that starts on an idle device (0.94 ms; 0.46 ms when calls
// follow one another, and here either way).  These calls allocate from a pool of their own, one per device, which
// keeps up to kScratchKeep bytes across synchronisations.  The pool orders reuse between streams and threads by
// itself; a destroyed context, an allocation that fails for want of memory (the driver's own allocations take what a
// pool keeps before they fail) and vpt_release_scratch give it back (scratch_trim).
#include "vpt_scratch.h"

#include <mutex>
#include "../../include/vpt_b200.h"

namespace vpt {
namespace {

constexpr unsigned long long kScratchKeep = 256ull << 20;  // a 1920 x 1080 SVGF call holds 180 MB
constexpr int kScratchDevices = 64;

std::mutex scratch_mutex;
cudaMemPool_t scratch_pools[kScratchDevices] = {};

// the current device's pool; nullptr where there is none (and create is false, or it cannot be made)
cudaMemPool_t scratch_pool(bool create) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kScratchDevices) return nullptr;
    std::lock_guard<std::mutex> lock(scratch_mutex);
    if (!scratch_pools[dev] && create) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        unsigned long long keep = kScratchKeep;
        if (cudaMemPoolCreate(&pool, &props) == cudaSuccess) {
            if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess)
                scratch_pools[dev] = pool;
            else
                cudaMemPoolDestroy(pool);
        }
        if (!scratch_pools[dev]) cudaGetLastError();  // the default pool serves; no error of the call
    }
    return scratch_pools[dev];
}

}  // namespace

cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s) {
    // a captured allocation belongs to its graph, whichever pool it names
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(s, &capture);
    if (e != cudaSuccess) return e;
    cudaMemPool_t pool = capture == cudaStreamCaptureStatusNone ? scratch_pool(true) : nullptr;
    if (!pool) return cudaMallocAsync(p, bytes, s);
    e = cudaMallocFromPoolAsync(p, bytes, pool, s);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    cudaMemPoolTrimTo(pool, 0);
    return cudaMallocFromPoolAsync(p, bytes, pool, s);
}

void scratch_trim() {
    if (cudaMemPool_t pool = scratch_pool(false)) cudaMemPoolTrimTo(pool, 0);
}

}  // namespace vpt

extern "C" VptStatus vpt_release_scratch(void) {
    vpt::scratch_trim();
    return VPT_OK;
}
