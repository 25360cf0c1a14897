// host_copy.cu -- device to host copies of whole fields.
//
// A copy into pageable memory goes through the driver's own staging and one
// host thread, which on freshly allocated arrays spends most of the time on
// page faults (2.7 GB/s on 9.4 MB).  Here the chunks of a large copy land in a
// small pinned buffer while a few threads move the chunks before them into the
// caller's array.  Measured with 16 cores, driver / here: two fresh arrays of
// 4.7 MB 3.3 / 1.1-1.4 ms, of 75 MB 32 / 11 ms; an array in use 4.7 MB 0.26 / 0.23
// ms, 75 MB 3.6 / 2.7 ms (four threads: 75 MB fresh 16 ms).
//
// The pinned buffer (16 MB) belongs to the process while any domain or fluid is
// alive: it is allocated by the first copy that needs it and freed with the
// last object.  One copy uses it at a time; another thread's copy meanwhile
// takes the driver's path.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>

#include "internal.h"

namespace sclbm {

namespace {
constexpr size_t CHUNK = size_t(512) << 10;
constexpr int SLOTS = 32;
constexpr int THREADS = 8; // at most, and half the cores
// smaller copies: the driver's path (1.6 MB: 0.14 ms, and 0.4 with threads to start)
constexpr size_t LEAST = size_t(3) << 20;

std::mutex g_mu; // the buffer and its events
char *g_buf = nullptr;
cudaEvent_t g_ev[SLOTS] = {};
int g_dev = -1;
std::atomic<long> g_objects{0};

void release_locked()
{
    for (auto &e : g_ev)
        if (e) {
            cudaEventDestroy(e);
            e = nullptr;
        }
    if (g_buf) cudaFreeHost(g_buf);
    g_buf = nullptr;
    g_dev = -1;
}

// the buffer and events of the current device; false: not to be had
bool acquire_locked(int dev)
{
    if (g_buf && g_dev == dev) return true;
    release_locked();
    bool ok = cudaHostAlloc((void **)&g_buf, CHUNK * SLOTS, cudaHostAllocPortable) == cudaSuccess;
    for (auto &e : g_ev) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    g_dev = dev;
    if (!ok) {
        cudaGetLastError();
        release_locked();
    }
    return ok;
}

cudaError_t plain_copy(void *dst, const void *src, size_t bytes, cudaStream_t s)
{
    const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s);
    return e != cudaSuccess ? e : cudaStreamSynchronize(s);
}

// One copy through the buffer: chunk i passes through slot i % SLOTS, its
// arrival marked by the slot's event; whoever has emptied a slot requests the
// chunk that comes next there.
struct Transfer {
    char *dst;
    const char *src;
    size_t bytes;
    cudaStream_t s;
    int dev, chunks;
    std::atomic<int> next{0}, requested{0}, error{cudaSuccess};

    size_t size(int i) const { return std::min(CHUNK, bytes - (size_t)i * CHUNK); }
    void fail(cudaError_t e)
    {
        int none = cudaSuccess;
        error.compare_exchange_strong(none, e);
    }
    void request(int i)
    {
        cudaError_t e = cudaMemcpyAsync(g_buf + (size_t)(i % SLOTS) * CHUNK, src + (size_t)i * CHUNK, size(i),
                                        cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaEventRecord(g_ev[i % SLOTS], s);
        if (e != cudaSuccess) fail(e);
    }
    void work()
    {
        for (int i; (i = next.fetch_add(1)) < chunks;) {
            // chunks are requested in order: a slot is emptied before the
            // request of the chunk after it, by a thread that waits for no one
            while (requested.load() <= i) {
                if (error.load() != cudaSuccess) return;
                std::this_thread::yield();
            }
            if (error.load() != cudaSuccess) return;
            const cudaError_t e = cudaEventSynchronize(g_ev[i % SLOTS]);
            if (e != cudaSuccess) return fail(e);
            std::memcpy(dst + (size_t)i * CHUNK, g_buf + (size_t)(i % SLOTS) * CHUNK, size(i));
            if (i + SLOTS < chunks) {
                while (requested.load() < i + SLOTS) { // in order
                    if (error.load() != cudaSuccess) return;
                    std::this_thread::yield();
                }
                request(i + SLOTS);
                requested.store(i + SLOTS + 1);
            }
        }
    }
};

cudaError_t bounced_copy(Transfer &t)
{
    const int first = std::min(t.chunks, SLOTS);
    for (int i = 0; i < first; ++i) t.request(i);
    t.requested.store(first);
    // whatever the stream had to do before the copy is waited for here, by one thread
    if (t.error.load() == cudaSuccess) {
        const cudaError_t e = cudaEventSynchronize(g_ev[0]);
        if (e != cudaSuccess) t.fail(e);
    }
    std::thread helpers[THREADS - 1];
    const int cores = (int)std::thread::hardware_concurrency();
    const int want = std::min({THREADS - 1, t.chunks - 1, std::max(0, cores / 2 - 1)});
    int n = 0;
    try {
        for (; n < want; ++n)
            helpers[n] = std::thread([&t] {
                const cudaError_t e = cudaSetDevice(t.dev);
                if (e != cudaSuccess) return t.fail(e);
                t.work();
            });
    } catch (const std::system_error &) {
        // fewer helpers: the others claim their chunks
    }
    t.work();
    for (int k = 0; k < n; ++k) helpers[k].join();
    const cudaError_t e = cudaStreamSynchronize(t.s); // after an error: no copy may still be under way
    return t.error.load() != cudaSuccess ? (cudaError_t)t.error.load() : e;
}
} // namespace

void host_copy_retain() { g_objects.fetch_add(1); }
void host_copy_release()
{
    if (g_objects.fetch_sub(1) != 1) return;
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_objects.load() == 0) release_locked();
}

bool host_copy_bounced(const void *dst, size_t bytes)
{
    cudaPointerAttributes at{};
    if (bytes < LEAST) return false;
    if (cudaPointerGetAttributes(&at, dst) == cudaSuccess) return at.type == cudaMemoryTypeUnregistered;
    cudaGetLastError();
    return false;
}

cudaError_t copy_to_host(void *dst, const void *src, size_t bytes, cudaStream_t s)
{
    if (!host_copy_bounced(dst, bytes)) return plain_copy(dst, src, bytes, s);
    int dev = 0;
    if (being_captured(s) || cudaGetDevice(&dev) != cudaSuccess) return plain_copy(dst, src, bytes, s);
    std::unique_lock<std::mutex> lk(g_mu, std::try_to_lock);
    if (!lk.owns_lock() || !acquire_locked(dev)) {
        if (lk.owns_lock()) lk.unlock();
        return plain_copy(dst, src, bytes, s);
    }
    Transfer t{(char *)dst, (const char *)src, bytes, s, dev, (int)((bytes + CHUNK - 1) / CHUNK)};
    return bounced_copy(t);
}

} // namespace sclbm
