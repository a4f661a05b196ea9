// csrc/part_sums.h with an allocator that fails at the n-th call: prints what the
// scratch claims to hold after each of a growth that fails at its first buffer, at
// its second, and one that succeeds (1: what it may, 0: more than it has).
#include <cstdio>
#include <cstdlib>
#include <type_traits>

#include "../vipp-nbody-bench_gb300/csrc/part_sums.h"

int main(int argc, char **argv) {
    if (argc == 7) {  // n, leaf, nsys, rows, bound, limit
        unsigned long long v[6];
        for (int i = 0; i < 6; ++i) v[i] = std::strtoull(argv[1 + i], nullptr, 10);
        std::printf("%u\n", gb::split_tiles_held(v[0], v[1], v[2], static_cast<unsigned>(v[3]), static_cast<unsigned>(v[4]), static_cast<unsigned>(v[5])));
        return 0;
    }
    int fail_at = 0, calls = 0;
    auto alloc = [&](auto *&p, std::size_t count) {
        std::free(p);
        p = nullptr;
        if (++calls == fail_at) return 2;  // out of memory
        using T = typename std::remove_reference<decltype(*p)>::type;
        p = static_cast<T *>(std::malloc(sizeof(T) * count));
        return 0;
    };
    for (int fail = 1; fail <= 3; ++fail) {
        gb::PartSums<double> s;
        fail_at = 0;
        bool ok = gb::resize(s, 40, 4, 40 * 10, alloc) == 0 && s.holds(40, 4) && s.holds(1, 1) && !s.holds(41, 4) && !s.holds(40, 5);
        fail_at = fail, calls = 0;
        const int e = gb::resize(s, 304, 10, 304 * 20, alloc);
        if (fail <= 2)  // neither the new size nor the old one, nor any other
            ok = ok && e == 2 && !s.holds(304, 10) && !s.holds(40, 4) && !s.holds(1, 1) && !s.holds(0, 0);
        else
            ok = ok && e == 0 && s.holds(304, 10);
        // the caller goes back to the smaller order: the buffers are made again
        fail_at = 0;
        if (!s.holds(40, 4)) ok = ok && gb::resize(s, 40, 4, 40 * 10, alloc) == 0;
        ok = ok && s.holds(40, 4) && s.part && s.cnt;
        std::printf("%d ", ok ? 1 : 0);
        std::free(s.part), std::free(s.cnt);
    }
    return 0;
}
