// host_pages.h -- the caller's result arrays, made ready for the copy that fills them.
//
// A result array is often fresh memory (numpy.empty, malloc): its pages do not exist yet, and a
// device-to-host copy then takes a fault through the IOMMU for each of them.  On a Grace host with
// 64 KB pages a copy of 67 MB took 2.6 ms into fresh pages and 0.41 ms into present ones (1 MB: 182
// and 28 us, 600 MB: 22 and 3.3 ms); the CPU makes pages at 33 GB/s on one thread, 100 GB/s on four,
// and more threads are slower again.  Callers first queue what the device still has to do and call
// this before they queue the copies, so that a busy device hides it altogether.
#pragma once

#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <atomic>
#include <initializer_list>
#include <exception>
#include <thread>

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23   // Linux 5.14; an older kernel refuses it and nothing is lost
#endif

namespace lbg {

struct HostRange {
    void *p;
    size_t bytes;
};

namespace host_pages_detail {

// Whether the range's pages are all present, or, of more than 64, 8 spread over it: making present pages
// ready costs as much as a fifth of the copy, so a buffer in use is left alone.
inline bool present(char *a, size_t len, size_t page)
{
    constexpr size_t ALL = 64, SAMPLES = 8;
    unsigned char v[ALL];
    const size_t pages = len / page;
    if (pages <= ALL) {   // one call
        if (mincore(a, len, v) != 0) return false;
        for (size_t k = 0; k < pages; ++k)
            if (!(v[k] & 1)) return false;
        return true;
    }
    for (size_t k = 0; k < pages; k += pages / SAMPLES)
        if (mincore(a + k * page, page, v) != 0 || !(v[0] & 1)) return false;
    return true;
}

}  // namespace host_pages_detail

// Null ranges are skipped, and memory that CUDA knows (registered, managed, device): only plain
// host memory is made ready.  Contents are kept.
inline void ready_pages(std::initializer_list<HostRange> ranges)
{
    constexpr size_t PIECE = 4u << 20, THREADED = 8u << 20;
    constexpr int MAX_RANGES = 8, HELPERS = 3;
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    struct {
        char *a;
        size_t len;
    } todo[MAX_RANGES];
    int n = 0;
    size_t total = 0;
    for (const HostRange &r : ranges) {
        if (!r.p || !r.bytes || n == MAX_RANGES) continue;
        char *a = (char *)((size_t)r.p / page * page);
        const size_t len = ((size_t)((char *)r.p + r.bytes - a) + page - 1) / page * page;
        // first, as a buffer in use is the common case and this the cheaper question (lbgpu_moments of 41^3:
        // 312 us without any, 328 with CUDA's for each of its four arrays)
        if (host_pages_detail::present(a, len, page)) continue;
        cudaPointerAttributes at;
        if (cudaPointerGetAttributes(&at, r.p) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        if (at.type != cudaMemoryTypeUnregistered) continue;
        todo[n++] = {a, len};
        total += len;
    }
    std::atomic<size_t> next{0};
    auto work = [&] {
        for (;;) {
            size_t at = next.fetch_add(PIECE);
            int k = 0;
            for (; k < n; ++k) {   // pieces are numbered range after range, each a whole number of them
                const size_t span = (todo[k].len + PIECE - 1) / PIECE * PIECE;
                if (at < span) break;
                at -= span;
            }
            if (k == n) return;
            madvise(todo[k].a + at, todo[k].len - at < PIECE ? todo[k].len - at : PIECE, MADV_POPULATE_WRITE);
        }
    };
    std::thread helper[HELPERS];
    if (total >= THREADED)
        for (std::thread &t : helper) {
            try {
                t = std::thread(work);
            } catch (const std::exception &) {   // no more threads, or no memory for one: this one does it
                break;
            }
        }
    work();
    for (std::thread &t : helper)
        if (t.joinable()) t.join();
}

}  // namespace lbg
