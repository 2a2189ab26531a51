// host_copy.h — the host's side of moving state vectors (solver.cu).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <thread>
#include <vector>

namespace pdipc {

// memcpy by a few threads when it is large.
inline void copy_host(double* dst, const double* src, size_t bytes) {
    constexpr size_t kPart = (size_t)1 << 20;  // below, a thread costs more than it saves
    const size_t parts = std::min<size_t>(6, bytes / kPart + 1);
    const size_t len = (bytes / parts + 63) / 64 * 64;
    auto part = [=](size_t k) {
        const size_t b = std::min(bytes, k * len), e = std::min(bytes, b + len);
        std::memcpy(reinterpret_cast<char*>(dst) + b, reinterpret_cast<const char*>(src) + b, e - b);
    };
    std::vector<std::thread> th;
    size_t started = 1;
    try {
        for (; started < parts; ++started) th.emplace_back(part, started);
    } catch (...) {  // no thread to be had: this one copies the rest
    }
    part(0);
    for (size_t k = started; k < parts; ++k) part(k);
    for (std::thread& t : th) t.join();
}

// Has every page of a buffer mapped before a copy engine writes it.  The bytes stay: a
// copy that then fails leaves the caller's data as it was.
inline void map_pages(void* buf, size_t bytes) {
    volatile char* p = static_cast<volatile char*>(buf);
    for (size_t b = 0; b < bytes; b += 4096) p[b] = p[b];
}

}  // namespace pdipc
