// Drives Readback (readback.hpp) over a CUDA runtime of host memory, so that its rules hold without a GPU:
// what a read does where memory cannot be pinned, from which device and threads it calls the runtime, and
// which destinations it copies into at once.  Argument: the rule to check.  Prints "ok" or what is wrong.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <set>
#include <string>
#include <thread>
#include <vector>

#include "celeris_internal.hpp"
#include "readback.hpp"

// ---- the runtime ----
static thread_local int t_device = 0;
static std::atomic<bool> g_refuse_pinned{false}, g_refuse_events{false};
static std::atomic<int> g_pinned{0}, g_wrong_device{0};
static int g_engine_device = 0;
static const char *g_known = nullptr, *g_known_end = nullptr;   // memory that the runtime knows
static cudaMemoryType g_known_type = cudaMemoryTypeHost;
static void on_device() { if (t_device != g_engine_device) ++g_wrong_device; }

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = t_device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { t_device = d; return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    if (g_refuse_pinned) return cudaErrorMemoryAllocation;
    ++g_pinned;
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { --g_pinned; std::free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    if (g_refuse_events) return cudaErrorMemoryAllocation;
    on_device();
    *e = reinterpret_cast<cudaEvent_t>(std::malloc(1));
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { on_device(); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    const char* c = static_cast<const char*>(p);
    std::memset(a, 0, sizeof(*a));
    a->type = c >= g_known && c < g_known_end ? g_known_type : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
}

using namespace cel;

static int fail(const char* what) { std::printf("%s\n", what); return 0; }

struct Source {   // what is read, and how it was asked for
    std::vector<char> data;
    std::atomic<int> wholes{0}, parts{0};
    std::mutex m;
    std::set<std::thread::id> threads;
    cudaError_t whole_error = cudaSuccess;
    explicit Source(size_t n) : data(n) {
        for (size_t i = 0; i < n; ++i) data[i] = char(i * 2654435761u >> 13);
    }
    void seen() {
        on_device();
        std::lock_guard<std::mutex> l(m);
        threads.insert(std::this_thread::get_id());
    }
    int read(Readback& rb, char* dst, cudaStream_t s, std::string& err) {
        return rb.read(
            dst, data.size(), s,
            [&](char* d) {
                seen();
                ++wholes;
                if (whole_error == cudaSuccess) std::memcpy(d, data.data(), data.size());
                return whole_error;
            },
            [&](size_t off, size_t n, char* slot) {
                seen();
                ++parts;
                std::memcpy(slot, data.data() + off, n);
                return cudaSuccess;
            },
            err);
    }
};

int main(int argc, char** argv) {
    const std::string rule = argc > 1 ? argv[1] : "";
    const size_t sizes[] = {16, READBACK_DIRECT, READBACK_DIRECT + 16, 3 * READBACK_SLOT + 48, size_t(17) << 20};
    const cudaStream_t own = reinterpret_cast<cudaStream_t>(0x1000);
    std::string err;
    for (const size_t n : sizes) {
        const bool small = n <= READBACK_DIRECT;
        Source src(n);
        std::vector<char> dst(n, 0);
        if (rule == "slots") {   // pageable destinations: small ones at once, others through slots
            Readback rb;
            if (src.read(rb, dst.data(), own, err) != CEL_OK || dst != src.data) return fail("wrong bytes");
            if (src.wholes != (small ? 1 : 0) || (src.parts == 0) != small) return fail("wrong route");
        } else if (rule == "refused") {   // no pinned memory, or no events: one pageable copy
            for (int what = 0; what < 2; ++what) {
                Readback rb;
                g_refuse_pinned = what == 0;
                g_refuse_events = what == 1;
                std::fill(dst.begin(), dst.end(), 0);
                if (src.read(rb, dst.data(), own, err) != CEL_OK) return fail("a read was refused");
                if (dst != src.data) return fail("wrong bytes");
            }
            g_refuse_pinned = g_refuse_events = false;
            Readback rb;   // and the slots again once there are some
            if (src.read(rb, dst.data(), own, err) != CEL_OK || (src.parts == 0) != small) return fail("slots not tried again");
        } else if (rule == "device") {   // a thread whose current device is another one than the engine's
            g_engine_device = t_device = 1;
            {
                Readback rb;
                t_device = 0;
                for (int k = 0; k < 2; ++k) {
                    if (src.read(rb, dst.data(), own, err) != CEL_OK || dst != src.data) return fail("wrong bytes");
                    if (t_device != 0) return fail("the caller's device was changed");
                }
            }
            if (g_wrong_device != 0) return fail("called on the wrong device");
        } else if (rule == "pinned") {   // memory that the runtime knows: one copy, as into any small destination
            g_known = dst.data();
            g_known_end = g_known + n;
            Readback rb;
            for (cudaMemoryType type : {cudaMemoryTypeHost, cudaMemoryTypeManaged}) {
                g_known_type = type;
                const int before = src.wholes;
                std::fill(dst.begin(), dst.end(), 0);
                if (src.read(rb, dst.data(), own, err) != CEL_OK || dst != src.data) return fail("wrong bytes");
                if (src.wholes != before + 1 || src.parts != 0) return fail("not copied into at once");
            }
            src.whole_error = cudaErrorInvalidValue;   // such as memory that is only partly registered: slots
            g_known_type = cudaMemoryTypeHost;
            std::fill(dst.begin(), dst.end(), 0);
            const int st = src.read(rb, dst.data(), own, err);
            if (!small && (st != CEL_OK || dst != src.data || src.parts == 0)) return fail("no second route");
            g_known_type = cudaMemoryTypeDevice;       // never written by the host
            if (src.read(rb, dst.data(), own, err) == CEL_OK) return fail("the host wrote into device memory");
        } else if (rule == "thread") {   // the per-thread stream is the calling thread's: no other may use it
            Readback rb;
            if (src.read(rb, dst.data(), cudaStreamPerThread, err) != CEL_OK || dst != src.data) return fail("wrong bytes");
            if (src.threads != std::set<std::thread::id>{std::this_thread::get_id()}) return fail("another thread's stream");
        } else {
            return fail("unknown rule");
        }
        if (g_pinned != 0) return fail("pinned blocks were left");
    }
    std::printf("ok\n");
    return 0;
}
