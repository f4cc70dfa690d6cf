// Copies of large results to pageable host memory.
#pragma once

#include <omp.h>

#include <algorithm>
#include <cstddef>
#include <cstring>

namespace ddm {

constexpr size_t kParallelCopyMin = 2u << 20;  // below, one thread copies as fast as it takes to wake others
constexpr size_t kParallelCopyPart = 512u << 10;

// memcpy by up to eight threads: the destination is often memory its process has not touched yet,
// and one thread spends most of the copy in its page faults.
inline void parallel_copy(void *dst, const void *src, size_t bytes) {
    const int threads = std::min(8, omp_get_max_threads());
    if (bytes < kParallelCopyMin || threads < 2 || omp_in_parallel()) {
        std::memcpy(dst, src, bytes);
        return;
    }
    const long long parts = static_cast<long long>((bytes + kParallelCopyPart - 1) / kParallelCopyPart);
#pragma omp parallel for num_threads(threads) schedule(static)
    for (long long i = 0; i < parts; i++) {
        const size_t at = static_cast<size_t>(i) * kParallelCopyPart;
        std::memcpy(static_cast<char *>(dst) + at, static_cast<const char *>(src) + at,
                    std::min(kParallelCopyPart, bytes - at));
    }
}

}  // namespace ddm
