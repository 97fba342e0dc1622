// column_copy.h -- a job's particle columns between host and device memory, and
// tables from host to device, written against the few calls of the CUDA runtime
// that they need, so that the order of copies and waits is checked on the CPU.
#pragma once

#include <cstddef>
#include <cstdint>
#include <initializer_list>
#include <vector>

namespace stg {

// The 21 columns of one particle set on the host, and its rows of `pitch`
// words on the device.
struct ColumnSet {
    void *cols[21];
    int64_t cnt;
    uint64_t *d;
    int64_t pitch;
};

// Straight between the two memories.  Columns at one distance, as the buffers
// lay them out, go in one copy: the host's work for each of 42 copies bounded
// a small set (push and collect of 1,000 particles from Python 257 -> 61 us
// with the columns read in one piece there), a staging block with its pages to
// fault in and its second pass over memory a large one (34 MB of
// element-by-element output 6.8 -> 0.19 ms).
template <class Api>
bool copy_columns(Api &api, const ColumnSet &set, bool to_device)
{
    if (set.cnt <= 0) return true;
    size_t const width = (size_t)set.cnt * 8, dev = (size_t)set.pitch * 8;
    uintptr_t const first = (uintptr_t)set.cols[0];
    size_t const apart = (uintptr_t)set.cols[1] - first;
    constexpr size_t kMaxPitch = 0x7fffffff;  // of a pitched copy
    bool even = (uintptr_t)set.cols[1] > first && apart >= width;
    for (int c = 2; c < 21; ++c) even = even && (uintptr_t)set.cols[c] == first + c * apart;
    bool const one = even && apart == width && dev == width;
    bool const pitched = even && apart <= kMaxPitch && dev <= kMaxPitch;
    size_t const bytes = one ? 21 * width : width;
    for (int c = 0; c < (one || pitched ? 1 : 21); ++c) {
        void *const host = set.cols[c], *const there = set.d + (size_t)c * set.pitch;
        void *const to = to_device ? there : host, *const from = to_device ? host : there;
        size_t const tp = to_device ? dev : apart, fp = to_device ? apart : dev;
        if (!(!one && pitched ? api.copy2d(to, tp, from, fp, width, 21)
                              : api.copy(to, from, bytes)))
            return false;
    }
    return true;
}

// Every set, and the wait for all of it: also after a failure (copies before
// it may be in flight), and also for copies that themselves return when the
// host memory is free again -- one from pageable memory has then been staged,
// not written, and the tracking kernels' stream does not wait for the stream it
// runs on.
template <class Api>
bool copy_sets(Api &api, const std::vector<ColumnSet> &sets, bool to_device)
{
    bool ok = true;
    for (const ColumnSet &s : sets) ok = ok && copy_columns(api, s, to_device);
    return api.wait() && ok;
}

struct BlockCopy {
    void *to;
    const void *from;
    size_t bytes;
};

// Blocks of words, and the wait for all of them.
template <class Api>
bool copy_blocks(Api &api, std::initializer_list<BlockCopy> blocks)
{
    bool ok = true;
    for (const BlockCopy &b : blocks)
        ok = ok && (b.bytes == 0 || api.copy(b.to, b.from, b.bytes));
    return api.wait() && ok;
}

}  // namespace stg
