// column_copy.h against a fake runtime on the CPU: a copy to the device only
// stages its source, and the data arrive when the stream is waited for.
// argv: layout, direction, failing call (-1: none).  Prints "ok", or what is
// wrong.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>

#include "column_copy.h"

using namespace stg;

struct Fake {
    bool to_device;
    int fail, calls = 0;
    std::vector<std::function<void()>> flight;

    bool copy2d(void *to, size_t tp, const void *from, size_t fp, size_t width, size_t rows)
    {
        if (calls++ == fail) return false;
        for (size_t r = 0; r < rows; ++r) {
            const char *src = (const char *)from + r * fp;
            char *dst = (char *)to + r * tp;
            std::vector<char> staged(src, src + width);
            auto land = [staged, dst] { std::memcpy(dst, staged.data(), staged.size()); };
            if (to_device)
                flight.push_back(land);
            else
                land();
        }
        return true;
    }
    bool copy(void *to, const void *from, size_t bytes)
    {
        return copy2d(to, bytes, from, bytes, bytes, 1);
    }
    bool wait()
    {
        for (auto &f : flight) f();
        flight.clear();
        return true;
    }
};

static int blocks(int fail)
{
    std::vector<uint64_t> const a(9, 3), b(5, 4);
    std::vector<uint64_t> dev(14, 0);
    Fake api{true, fail};
    bool const done =
        copy_blocks(api, {{dev.data(), a.data(), 72}, {nullptr, nullptr, 0}, {&dev[9], b.data(), 40}});
    if (!api.flight.empty()) return puts("copies in flight after the return"), 0;
    if (done != (fail < 0 || fail >= api.calls)) return puts("a failure was not reported"), 0;
    for (int i = 0; done && i < 14; ++i)
        if (dev[i] != (i < 9 ? 3u : 4u)) return printf("word %d\n", i), 0;
    return puts("ok"), 0;
}

int main(int argc, char **argv)
{
    if (argc < 4) return 2;
    if (!strcmp(argv[1], "blocks")) return blocks(atoi(argv[3]));
    bool const to_device = !strcmp(argv[2], "up");
    int const fail = atoi(argv[3]);
    // two sets in one block on the device; the host's columns back to back, at
    // a common distance, or anywhere
    int64_t const cnt[2] = {7, 0 == strcmp(argv[1], "single") ? 0 : 5}, total = cnt[0] + cnt[1];
    std::vector<uint64_t> dev(21 * total, 1), host(2 * 21 * 64, 2);
    std::vector<ColumnSet> sets;
    for (int k = 0; k < 2; ++k) {
        ColumnSet s{{}, cnt[k], dev.data() + (k ? cnt[0] : 0), total};
        for (int c = 0; c < 21; ++c) {
            int64_t at = c * cnt[k];
            if (!strcmp(argv[1], "apart")) at = c * 40;
            if (!strcmp(argv[1], "uneven")) at = 64 * ((5 * c) % 21) + c;
            s.cols[c] = &host[k * 21 * 64 + at];
        }
        sets.push_back(s);
    }
    auto host_at = [&](int k, int c, int64_t i) -> uint64_t & {
        return ((uint64_t *)sets[k].cols[c])[i];
    };
    auto dev_at = [&](int k, int c, int64_t i) -> uint64_t & { return sets[k].d[c * total + i]; };
    for (int k = 0; k < 2; ++k)
        for (int c = 0; c < 21; ++c)
            for (int64_t i = 0; i < cnt[k]; ++i)
                (to_device ? host_at(k, c, i) : dev_at(k, c, i)) = 1000 * (k + 1) + 21 * i + c;
    Fake api{to_device, fail};
    bool const done = copy_sets(api, sets, to_device);
    if (!api.flight.empty()) return puts("copies in flight after the return"), 0;
    if (done != (fail < 0 || fail >= api.calls)) return puts("a failure was not reported"), 0;
    for (int k = 0; done && k < 2; ++k)
        for (int c = 0; c < 21; ++c)
            for (int64_t i = 0; i < cnt[k]; ++i)
                if (host_at(k, c, i) != dev_at(k, c, i) ||
                    host_at(k, c, i) != (uint64_t)(1000 * (k + 1) + 21 * i + c))
                    return printf("set %d column %d particle %d\n", k, c, (int)i), 0;
    return puts("ok"), 0;
}
