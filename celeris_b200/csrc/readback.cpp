// Reads of whole textures into the caller's (pageable) host memory.
//
// What bounds a read is the host: the planes used to come back one pageable copy each (24 bytes a
// texel in the compensated form, through the driver's single staging thread) and a scalar loop
// interleaved them into fresh, still unmapped memory.  Here a kernel forms the 16-byte texels on the
// device and writes them straight into pinned slots over the bus, and the slots are copied into the
// caller's memory while the next ones fill; for large reads several threads do that, since the copy
// and the page faults of the destination take longer than the bus (16.9 MB into fresh memory: one
// thread 3.1 ms, six 2.1).  Up to 1 MB the texels are formed in device memory and copied at once: a
// first read must not wait for memory to be pinned (2.3 ms).
// Measured, compensated form: 2052 x 2052 texels 40 -> 5.5 ms, 1028 x 1028 7.9 -> 2.1, 516 x 68 0.30 ->
// 0.16, 28 members of 256^2 .. 2048 x 512 126 -> 34.
#include "readback.hpp"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

#include "celeris_internal.hpp"

namespace cel {

// ---- the pool of pinned blocks ------------------------------------------------------------------
namespace {

constexpr size_t BLOCK = READBACK_SLOT * READBACK_SLOTS;
std::mutex g_pool_mutex;                 // guards the three below
std::vector<char*> g_pool;               // free blocks
int g_users = 0;                         // live Readbacks

char* take_block(cudaError_t& e) {
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        if (!g_pool.empty()) {
            char* p = g_pool.back();
            g_pool.pop_back();
            return p;
        }
    }
    void* p = nullptr;
    e = cudaHostAlloc(&p, BLOCK, cudaHostAllocMapped | cudaHostAllocPortable);   // any device may write it
    return e == cudaSuccess ? static_cast<char*>(p) : nullptr;
}

void give_block(char* p) {
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        if (g_pool.size() < READBACK_CACHED) {   // (room reserved by the first Readback: no throw)
            g_pool.push_back(p);
            return;
        }
    }
    cudaFreeHost(p);
}

// The owner's device for the length of a read: launches and events need it current (a new thread starts on
// device 0).
class OnDevice {
public:
    explicit OnDevice(int dev) {
        if (dev >= 0 && cudaGetDevice(&before_) == cudaSuccess && before_ != dev) moved_ = cudaSetDevice(dev) == cudaSuccess;
    }
    OnDevice(const OnDevice&) = delete;
    OnDevice& operator=(const OnDevice&) = delete;
    ~OnDevice() {
        if (moved_) cudaSetDevice(before_);
    }

private:
    int before_ = 0;
    bool moved_ = false;
};

}  // namespace

Readback::Readback() {
    if (cudaGetDevice(&dev_) != cudaSuccess) dev_ = -1;
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    g_pool.reserve(READBACK_CACHED);
    ++g_users;
}

Readback::~Readback() {
    for (cudaEvent_t e : ev_)
        if (e) cudaEventDestroy(e);
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    if (--g_users > 0) return;
    for (char* p : g_pool) cudaFreeHost(p);
    g_pool.clear();
}

int Readback::read_whole(char* dst, cudaStream_t s, const std::function<cudaError_t(char* dst)>& whole, std::string& err) {
    cudaError_t e = whole(dst);
    const cudaError_t w = cudaStreamSynchronize(s);   // also after an error: nothing may still write into dst
    if (e == cudaSuccess) e = w;
    if (e == cudaSuccess) return CEL_OK;
    err = std::string("read-back: ") + cudaGetErrorString(e);
    return CEL_ERR_CUDA;
}

int Readback::read(void* dst, size_t bytes, cudaStream_t s, const std::function<cudaError_t(char* dst)>& whole,
                   const std::function<cudaError_t(size_t offset, size_t n, char* slot)>& part, std::string& err) {
    if (bytes == 0) return CEL_OK;
    const OnDevice on(dev_);
    if (bytes <= READBACK_DIRECT) return read_whole(static_cast<char*>(dst), s, whole, err);
    // Memory that the runtime knows is copied into at once.  Pinned by the caller it takes the bus's rate, and
    // the slots' host copy only adds to that (plain form, 2052 x 2052 texels 2.6 -> 1.2 ms, 704 x 504 0.52 -> 0.11);
    // the host must not write into device memory.
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, dst) != cudaSuccess) {
        (void)cudaGetLastError();
        at.type = cudaMemoryTypeUnregistered;
    }
    if (at.type != cudaMemoryTypeUnregistered) {
        const int st = read_whole(static_cast<char*>(dst), s, whole, err);
        if (st == CEL_OK || at.type == cudaMemoryTypeDevice) return st;
        (void)cudaGetLastError();   // such as memory that is registered in part: through slots
    }
    const size_t chunk = std::min(READBACK_SLOT, bytes);
    const size_t chunks = (bytes + chunk - 1) / chunk;
    // starting a thread takes as long as copying a few hundred kB
    int workers = int(std::min<size_t>(READBACK_WORKERS, bytes / READBACK_SHARE));
    workers = std::max(1, std::min(workers, int(std::thread::hardware_concurrency())));
    if (s == cudaStreamPerThread) workers = 1;   // in a helper thread this name is another stream, which waits for nothing
    cudaError_t first = cudaSuccess;
    for (int k = 0; k < READBACK_SLOTS && first == cudaSuccess; ++k)
        if (!ev_[k]) first = cudaEventCreateWithFlags(&ev_[k], cudaEventDisableTiming);
    int dev = 0;   // for the helper threads
    if (first == cudaSuccess) first = cudaGetDevice(&dev);
    char* const block = first == cudaSuccess ? take_block(first) : nullptr;
    if (!block) {   // no slots (a limit on pinned memory): one copy needs none
        (void)cudaGetLastError();
        return read_whole(static_cast<char*>(dst), s, whole, err);
    }
    std::atomic<int> failed{int(cudaSuccess)};
    // worker w takes chunks w, w + workers, ... through slots 2w and 2w + 1: two in flight
    auto work = [&](int w, int nw) {
        cudaError_t e = cudaSetDevice(dev);
        auto put = [&](size_t c, int slot) -> cudaError_t {
            const size_t off = c * chunk;
            cudaError_t r = part(off, std::min(chunk, bytes - off), block + size_t(slot) * READBACK_SLOT);
            return r == cudaSuccess ? cudaEventRecord(ev_[slot], s) : r;
        };
        size_t next = size_t(w);
        for (int q = 0; q < 2 && e == cudaSuccess && next < chunks; ++q, next += size_t(nw)) e = put(next, 2 * w + q);
        int q = 0;
        for (size_t c = size_t(w); c < chunks && e == cudaSuccess; c += size_t(nw), q ^= 1) {
            const int slot = 2 * w + q;
            e = cudaEventSynchronize(ev_[slot]);
            if (e != cudaSuccess) break;
            const size_t off = c * chunk;
            std::memcpy(static_cast<char*>(dst) + off, block + size_t(slot) * READBACK_SLOT, std::min(chunk, bytes - off));
            if (next < chunks) { e = put(next, slot); next += size_t(nw); }
        }
        if (e != cudaSuccess) failed = int(e);
    };
    if (workers == 1) {
        work(0, 1);
    } else {
        std::vector<std::thread> team;
        int started = 1;
        try {
            team.reserve(size_t(workers));
            for (; started < workers; ++started) team.emplace_back(work, started, workers);
        } catch (const std::exception&) {   // no more threads: this one takes the shares that are left
        }
        work(0, workers);
        for (int w = started; w < workers; ++w) work(w, workers);
        for (std::thread& t : team) t.join();
    }
    if (failed != int(cudaSuccess)) (void)cudaStreamSynchronize(s);   // nothing may still write into the slots
    give_block(block);
    if (failed != int(cudaSuccess)) {
        err = std::string("read-back: ") + cudaGetErrorString(cudaError_t(failed.load()));
        return CEL_ERR_CUDA;
    }
    return CEL_OK;
}

}  // namespace cel
