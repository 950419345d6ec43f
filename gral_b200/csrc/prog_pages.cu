// prog_pages.cu -- first touch of a call's result arrays (prog_pages.cuh).
#include "prog_pages.cuh"

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <thread>
#include <vector>

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23     // Linux 5.14; older kernels refuse it and nothing happens
#endif

namespace gral {

namespace {

constexpr size_t kPiece = (size_t)512 << 10;   // of one request: a thread's share of the work
constexpr size_t kArray = (size_t)1 << 20, kTotal = (size_t)4 << 20;
constexpr int kThreads = 4;

// whether most of 8 pages spread over [b, e) are not there yet
bool untouched(char *b, char *e, size_t page) {
    int out = 0;
    for (int q = 0; q < 8; ++q) {
        char *p = b + (size_t)(e - b) / page * q / 8 * page;
        unsigned char there = 1;
        if (mincore(p, page, &there) != 0) return false;
        out += !(there & 1);
    }
    return out > 4;
}

}  // namespace

void first_touch(std::initializer_list<HostRange> ranges) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    std::vector<HostRange> pieces;
    size_t total = 0;
    for (const HostRange &r : ranges) {
        if (!r.p || r.bytes < kArray) continue;
        // whole pages inside the array
        char *b = (char *)(((uintptr_t)r.p + page - 1) / page * page), *e = (char *)(((uintptr_t)r.p + r.bytes) / page * page);
        if (!untouched(b, e, page)) continue;
        total += (size_t)(e - b);
        for (char *p = b; p < e; p += kPiece) pieces.push_back(HostRange{p, std::min(kPiece, (size_t)(e - p))});
    }
    if (total < kTotal) return;
    std::atomic<size_t> next{0};
    auto work = [&] {
        for (size_t q; (q = next.fetch_add(1)) < pieces.size();)
            if (madvise(pieces[q].p, pieces[q].bytes, MADV_POPULATE_WRITE) != 0) return;
    };
    const int threads = std::min(kThreads, (int)std::max(1u, std::thread::hardware_concurrency() / 2));
    std::vector<std::thread> pool;
    pool.reserve(threads);
    for (int t = 1; t < threads; ++t) {
        try {
            pool.emplace_back(work);
        } catch (...) {      // no more threads: those there are do the work
            break;
        }
    }
    work();
    for (auto &t : pool) t.join();
}

}  // namespace gral
