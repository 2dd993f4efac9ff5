// Host test shim: a large result's download (simple3.0_b200/csrc/download.h, the same source the library
// compiles) over a device whose copies land only when they are waited for.
#include "download.h"

#include <vector>

namespace {
struct FakeDev {
    const char *src;
    char *dst;
    size_t bytes;
    bool page_locked;
    int npieces, fail_copy;   // pinned buffers to be had; the copy (from 0) that fails, or -1
    int copies = 0, direct = 0;
    struct Copy { char *to; size_t off, n; };
    std::vector<Copy> flight;             // since the last mark
    std::vector<Copy> held[2];
    std::vector<char> buf[2];

    bool pageable() const { return !page_locked; }
    char *piece(int i)
    {
        if (i >= npieces) return nullptr;
        buf[i].resize(pftcc::DL_PIECE);
        return buf[i].data();
    }
    int copy(void *to, size_t off, size_t n)
    {
        if (copies++ == fail_copy) return 7;
        char *t = static_cast<char *>(to);
        direct += t >= dst && t < dst + bytes;
        flight.push_back({t, off, n});
        return 0;
    }
    int mark(int i) { held[i].swap(flight); flight.clear(); return 0; }
    void land(std::vector<Copy> &v)
    {
        for (const Copy &c : v) std::memcpy(c.to, src + c.off, c.n);
        v.clear();
    }
    int wait(int i) { land(held[i]); return 0; }
    int sync() { land(flight); return 0; }
};
}  // namespace

extern "C" int download_run(const char *src, char *dst, size_t bytes, int page_locked, int npieces, int fail_copy, int *copies,
                            int *direct)
{
    FakeDev d{src, dst, bytes, page_locked != 0, npieces, fail_copy};
    const int st = pftcc::download(d, dst, bytes);
    *copies = d.copies;
    *direct = d.direct;
    return st;
}
