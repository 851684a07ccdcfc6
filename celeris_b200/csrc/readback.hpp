// Device arrays to caller-owned host memory in the public RGBA32F layout.
#pragma once

#include <cuda_runtime.h>

#include <functional>
#include <string>

namespace cel {

// What one output texel is made of: planes of pitch P (hi, lo: w, hu, hv), or the aux pair plane.
enum PackMode { PACK_SUM, PACK_HI, PACK_LO, PACK_AUX };
struct PackArgs {
    const float* hi[3];
    const float* lo[3];      // null without low words
    const float2* aux;
    int NX, P;
    int mode;                // PackMode
};
// Writes texels [first, first + count) of the NX-wide texture to out, as float4, on stream s.
cudaError_t launch_pack(const PackArgs& a, size_t first, size_t count, float4* out, cudaStream_t s);

// Reads into pageable memory through pinned slots.  The slots come from a pool shared by every engine
// and lane of the process (pinning memory takes milliseconds): a read takes a block for its duration,
// READBACK_CACHED blocks at most wait for the next one, and they are freed with the last Readback.  The
// pool may be used from several threads; one Readback, like its owner, from one at a time.
constexpr size_t READBACK_DIRECT = size_t(1) << 20;   // reads up to here are one pageable copy
constexpr size_t READBACK_SLOT = size_t(512) << 10;
constexpr size_t READBACK_SHARE = size_t(2) << 20;    // bytes that pay for one more thread
constexpr int READBACK_WORKERS = 6;
constexpr int READBACK_SLOTS = 2 * READBACK_WORKERS;
constexpr int READBACK_CACHED = 4;
class Readback {
public:
    Readback();   // on its owner's device, where every read runs, whichever device is current in the caller's thread
    Readback(const Readback&) = delete;
    Readback& operator=(const Readback&) = delete;
    ~Readback();
    // Fills dst[0, bytes) and waits.  part(offset, n, slot) puts the work that fills slot[0, n) with the
    // bytes from `offset` on the stream; it may be called from helper threads.  whole(dst) puts work and one
    // copy there that fill dst at once: for reads up to READBACK_DIRECT, and where there are no slots to be
    // had (a limit on pinned memory).  Returns a CEL_* status.
    int read(void* dst, size_t bytes, cudaStream_t s, const std::function<cudaError_t(char* dst)>& whole,
             const std::function<cudaError_t(size_t offset, size_t n, char* slot)>& part, std::string& err);

private:
    int read_whole(char* dst, cudaStream_t s, const std::function<cudaError_t(char* dst)>& whole, std::string& err);
    int dev_ = -1;                          // the owner's device
    cudaEvent_t ev_[READBACK_SLOTS] = {};   // created by the first read through slots
};

}  // namespace cel
