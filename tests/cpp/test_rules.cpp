// Host-side rules of magpy_gb300/csrc/rules.hpp on sizes; exits non-zero at the
// first that fails.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include "rules.hpp"

using namespace magpy;

#define CHECK(x)                                             \
    do {                                                     \
        if (!(x)) {                                          \
            std::fprintf(stderr, "line %d: %s\n", __LINE__, #x); \
            std::exit(1);                                    \
        }                                                    \
    } while (0)

static void adjoint()
{
    const size_t GB = (size_t)1 << 30, P = 27 * 64, K = 20000, C = 256;  // 1.24e9 bytes in all
    CHECK(adjoint_keep(K, C, P, 200 * GB) == AdjointKeep::whole);
    CHECK(adjoint_keep(K, C, P, 19 * GB) == AdjointKeep::whole);
    CHECK(adjoint_keep(K, C, P, 18 * GB) == AdjointKeep::segment);  // 16 times 1.16 GiB
    CHECK(adjoint_keep(K, C, P, GB / 2) == AdjointKeep::segment);
    CHECK(adjoint_keep(K, C, P, GB / 8) == AdjointKeep::none);
    CHECK(adjoint_keep(K, C, P, 0) == AdjointKeep::none);
    // at most 4 GiB whatever is free, at most a sixteenth of what is free
    for (size_t free_gb : {1, 3, 17, 64, 65, 280})
        for (size_t k = 1; k < 3000000; k = k * 3 / 2 + 1) {
            const size_t bytes = 36 * k * P;
            if (adjoint_keep(k, C, P, free_gb * GB) == AdjointKeep::whole)
                CHECK(bytes <= 4 * GB && bytes <= free_gb * GB / 16);
        }
    // no size product wraps
    CHECK(adjoint_keep((size_t)1 << 32, (size_t)1 << 62, (size_t)1 << 40, 280 * GB) ==
          AdjointKeep::none);
    CHECK(adjoint_keep((size_t)1 << 32, 1, 1024, 280 * GB) == AdjointKeep::segment);
    CHECK(adjoint_keep(100, 10, 0, GB) == AdjointKeep::whole);  // no members
}

int main()
{
    adjoint();
    std::puts("rules ok");
    return 0;
}
