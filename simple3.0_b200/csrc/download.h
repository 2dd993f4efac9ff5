// download.h -- a large result's way into the caller's host memory (corr_all, corr_all_prec), over the
// few device calls it needs (Dev), so that the route and the order are tested without a GPU.
//
// Page-locked memory takes one direct copy.  A large result into pageable memory goes in pieces through
// two pinned buffers, the next piece on its way while this one is copied out by a few threads (which
// also take the page faults of fresh memory side by side): one pageable copy of 51 MB took 10.7 ms of
// corr_all's 13.2, this takes 4.5.  Below 32 MiB the plain copy is the faster: the allocator then gives back
// pages that are already there, and there are no faults to share.  corr_all_prec into a new array, ms, through
// the pieces and plain: 8 MiB 1.8 and 1.4, 16 MiB 2.8 and 2.5, 24 MiB 4.2 and 3.5, but 32 MiB 3.8 and 8.0, 64 MiB
// 7.8 and 15.  The plain copy also serves where no pinned memory is to be had.
//
//   Dev::pageable()                false where the destination is page-locked (or not host memory)
//   Dev::piece(i)                  pinned buffer i of 2, DL_PIECE bytes; null where there is none
//   Dev::copy(dst, offset, n)      the asynchronous copy of n bytes of the result; 0 or an error
//   Dev::mark(i), Dev::wait(i)     buffer i's last copy recorded, and waited for
//   Dev::sync()                    every copy waited for
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <system_error>
#include <thread>

namespace pftcc {

constexpr size_t DL_PIECE = 4u << 20;
constexpr size_t DL_MIN = 32u << 20;   // the smallest result that goes in pieces
constexpr int DL_THREADS = 4;

inline void copy_out(char *dst, const char *src, size_t bytes)
{
    std::thread th[DL_THREADS - 1];
    const size_t part = (bytes / DL_THREADS + 4095) & ~size_t(4095);
    int started = 0;
    try {
        for (; started < DL_THREADS - 1 && (started + 1) * part < bytes; ++started) {
            const size_t o = (started + 1) * part;
            th[started] = std::thread([=] { std::memcpy(dst + o, src + o, std::min(part, bytes - o)); });
        }
    } catch (const std::system_error &) {   // no more threads: the rest here
    }
    std::memcpy(dst, src, std::min(part, bytes));
    const size_t o = (size_t)(started + 1) * part;
    if (o < bytes) std::memcpy(dst + o, src + o, bytes - o);
    for (int i = 0; i < started; ++i) th[i].join();
}

template <class Dev> int download(Dev &dev, char *dst, size_t bytes)
{
    int st;
    if (bytes < DL_MIN || !dev.pageable() || !dev.piece(0) || !dev.piece(1)) {
        if ((st = dev.copy(dst, 0, bytes))) return st;
        return dev.sync();
    }
    const size_t n = (bytes + DL_PIECE - 1) / DL_PIECE;
    auto size = [&](size_t i) { return std::min(DL_PIECE, bytes - i * DL_PIECE); };
    for (size_t i = 0; i <= n; ++i) {
        // the buffer was copied out two pieces ago
        if (i < n && ((st = dev.copy(dev.piece(i & 1), i * DL_PIECE, size(i))) || (st = dev.mark(i & 1)))) return st;
        if (i == 0) continue;
        if ((st = dev.wait((i - 1) & 1))) return st;
        copy_out(dst + (i - 1) * DL_PIECE, dev.piece((i - 1) & 1), size(i - 1));
    }
    return 0;
}

}  // namespace pftcc
