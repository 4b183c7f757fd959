// parallel_for (bvh_build.h) covers every index exactly once, on the sizes around its piece
// length and thread count (test infrastructure, run by tests/test_parallel_for.py).
#include <atomic>
#include <cstdio>
#include <memory>

#include "bvh_build.h"

int main() {
    int failures = 0;
    for (size_t n : {(size_t)0, (size_t)1, (size_t)8191, (size_t)8192, (size_t)16383, (size_t)16384, (size_t)16385,
                     (size_t)65535, (size_t)65537, (size_t)100003, (size_t)1000000}) {
        std::unique_ptr<std::atomic<int>[]> seen(new std::atomic<int>[n + 1]());
        ftb::parallel_for(n, [&](size_t a, size_t b) {
            for (size_t i = a; i < b; ++i) seen[i].fetch_add(1);
        });
        bool ok = seen[n] == 0;
        for (size_t i = 0; i < n; ++i) ok = ok && seen[i] == 1;
        std::printf("n=%zu: %s\n", n, ok ? "ok" : "wrong");
        failures += ok ? 0 : 1;
    }
    return failures ? 1 : 0;
}
