// host_copy.cu -- device to host copies of whole fields.
//
// A freshly allocated array has no pages behind it: copied into as it is, the
// driver's one copying thread takes a page fault every 4 KB, after the stream
// has done its work (2.0 GB/s, against 19 into an array in use).  Here its pages
// are asked for first, while the stream still works, by up to four threads for
// larger arrays; the copy itself is the driver's.  Nothing is kept between
// calls: a pinned buffer that a copy passes through costs 20 ms to allocate,
// which a program that reads one field of an object never gets back.
//
// Measured with 16 cores, ms without / with (alone; behind steps that take
// longer than the pages): 4.7 MB 2.3 / 1.5; 2.3 / 0.29, 9.7 MB 4.8 / 2.5; 4.7 /
// 0.84, 75 MB 36.9 / 11.8.  An array in use, 4.7 MB: 0.27 / 0.27.
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstdint>
#include <exception>
#include <thread>

#include "internal.h"

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23 // Linux 5.14
#endif

namespace sclbm {

namespace {
constexpr size_t LEAST = size_t(3) << 20;  // smaller arrays: malloc hands out pages in use
constexpr size_t SHARE = size_t(4) << 20;  // per thread; starting one takes as long as 0.3 MB of pages
constexpr int THREADS = 4;                 // eight were slower (75 MB 15.9 ms)

// whether some of the page-aligned range has no pages yet, by five of them
bool pages_missing(char *a, size_t len, size_t page)
{
    for (int k = 0; k < 5; ++k) {
        unsigned char in = 1;
        const size_t at = (len / page - 1) * k / 4 * page;
        if (mincore(a + at, page, &in) == 0 && !(in & 1)) return true;
    }
    return false;
}
} // namespace

void host_pages_in(void *dst, size_t bytes)
{
    cudaPointerAttributes at{};
    if (bytes < LEAST) return;
    if (cudaPointerGetAttributes(&at, dst) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    if (at.type != cudaMemoryTypeUnregistered) return;
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    const uintptr_t first = ((uintptr_t)dst + page - 1) / page * page, end = ((uintptr_t)dst + bytes) / page * page;
    if (end <= first) return;
    char *const a = (char *)first;
    const size_t len = end - first;
    if (!pages_missing(a, len, page)) return;
    const int cores = (int)std::thread::hardware_concurrency();
    const int n = std::max(1, std::min({THREADS, cores / 2, (int)std::min<size_t>(len / SHARE, THREADS)}));
    // a failure (an older kernel, an odd mapping) leaves the faults to the copy
    auto part = [=](int k) {
        const size_t b = len / page * k / n * page, e = len / page * (k + 1) / n * page;
        madvise(a + b, e - b, MADV_POPULATE_WRITE);
    };
    std::thread helpers[THREADS];
    int k = 1;
    try {
        for (; k < n; ++k) helpers[k] = std::thread(part, k);
    } catch (const std::exception &) { // no more threads: the copy takes these faults
    }
    part(0);
    for (int j = 1; j < k; ++j) helpers[j].join();
}

cudaError_t copy_to_host(void *dst, const void *src, size_t bytes, cudaStream_t s)
{
    host_pages_in(dst, bytes);
    const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s);
    return e != cudaSuccess ? e : cudaStreamSynchronize(s);
}

} // namespace sclbm
