// Host-side check of the wide nodes' child codes (test infrastructure, built and run by
// tests/test_node_codes.py).  For trees of the host builder over seeded box sets, every child
// slot's code byte must name the same child as its meta byte: the entry the traversal forms,
// base of the kind + (code & 127), equals the node index, or the leaf's first record and
// count, that the meta byte describes; and the rows of planes sit on 32-byte sectors.
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <random>
#include <string>
#include <vector>

#include "bvh_build.h"

namespace ftb {
// the device builder is not part of this check
bool build_wide_lbvh_device(const std::vector<Box>&, int, int, WideBvh&, std::string& err) {
    err = "no device";
    return false;
}
}  // namespace ftb

using namespace ftb;

static uint32_t entry_of_code(const FNode& n, int k) {
    const uint32_t c = n.code[k];
    return ((c & 0x80u) ? (0x80000000u | (n.prim_base << 2)) : n.child_base) + (c & 0x7fu);
}
static uint32_t entry_of_meta(const FNode& n, int k) {
    const uint32_t m = n.meta[k];
    if ((m >> 5) == FNODE_INNER) return n.child_base + (m & 31u);
    return 0x80000000u | ((n.prim_base + (m & 31u)) << 2) | ((m >> 5) - 1u);
}

int main() {
    static_assert(offsetof(FNode, lo) % 32 == 0 && offsetof(FNode, hi) % 32 == 0 && sizeof(FNode) % 32 == 0, "rows");
    std::mt19937_64 rng(777);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    int failures = 0;
    for (int n : {1, 2, 7, 8, 9, 31, 33, 257, 20000}) {
        std::vector<Box> boxes((size_t)n);
        for (Box& b : boxes)
            for (int a = 0; a < 3; ++a) {
                const double c = u(rng), h = 0.02 * u(rng) * u(rng);
                b.lo[a] = c - h;
                b.hi[a] = c + h;
            }
        WideBvh b;
        std::string err;
        bool ok = build_wide_bvh(boxes, std::ldexp(1.0, -18), b, err) && validate_wide_bvh(b, n, err);
        size_t leaves = 0, inner = 0;
        if (ok) {
            const std::vector<FNode> f = widen_nodes(b);
            for (const FNode& x : f)
                for (int k = 0; k < FTB_WIDTH; ++k) {
                    if (!x.meta[k]) continue;
                    ((x.meta[k] >> 5) == FNODE_INNER ? inner : leaves)++;
                    if (entry_of_code(x, k) != entry_of_meta(x, k)) ok = false;
                }
        }
        std::printf("n=%d inner=%zu leaves=%zu: %s\n", n, inner, leaves, ok ? "ok" : "differs");
        failures += ok ? 0 : 1;
    }
    return failures ? 1 : 0;
}
