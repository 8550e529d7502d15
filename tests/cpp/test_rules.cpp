// Host-side rules of magpy_gb300/csrc/rules.hpp on sizes; exits non-zero at the
// first that fails.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>
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
    CHECK(adjoint_keep(K, 2 * C, 16 * P, 0) == AdjointKeep::none);
    // up to 64 MiB without asking
    CHECK(adjoint_keep(K, C, P, 0) == AdjointKeep::segment);
    CHECK(adjoint_keep(1078, C, P, 0) == AdjointKeep::whole);
    CHECK(adjoint_keep(1079, C, P, 0) == AdjointKeep::segment);
    // at most 4 GiB whatever is free, at most a sixteenth of what is free
    for (size_t free_gb : {1, 3, 17, 64, 65, 280})
        for (size_t k = 1; k < 3000000; k = k * 3 / 2 + 1) {
            const size_t bytes = 36 * k * P;
            if (adjoint_keep(k, C, P, free_gb * GB) == AdjointKeep::whole)
                CHECK(bytes <= 4 * GB && bytes <= std::max(GB / 16, free_gb * GB / 16));
        }
    // no size product wraps
    CHECK(adjoint_keep((size_t)1 << 32, (size_t)1 << 62, (size_t)1 << 40, 280 * GB) ==
          AdjointKeep::none);
    CHECK(adjoint_keep((size_t)1 << 32, 1, 1024, 280 * GB) == AdjointKeep::segment);
    CHECK(adjoint_keep(100, 10, 0, GB) == AdjointKeep::whole);  // no members
}

// Whatever the SM count: no wave of one-CTA-an-SM blocks more than 32 members a
// CTA need, and fewer members only while that holds.
static void tensor_core_members()
{
    for (int sms : {1, 76, 132, 148, 152, 160})
        for (int64_t E = 1; E < 100000; E += 1 + E / 37) {
            const int m = tc_members(E, sms);
            const auto ctas = [&](int k) { return (E + k - 1) / k; };
            const auto waves = [&](int k) { return (ctas(k) + sms - 1) / sms; };
            CHECK(m >= 8 && m <= 32 && m % 4 == 0);
            CHECK(waves(m) == waves(32));
            if (m > 8) CHECK(waves(m - 4) > waves(32));
        }
    CHECK(tc_members(4096, 152) == 28 && tc_members(4096, 148) == 28);
    CHECK(tc_members(28 * 152, 152) == 28 && tc_members(28 * 152, 148) == 32);
}

// While a batch is small enough every warp has a sub-partition; then only
// particles far above the mean get five lanes.
static void two_state_lanes()
{
    for (int sms : {76, 148, 152})
        for (int64_t E : {1, 6, 1000, 8192, 17000, 19456, 65536}) {
            const std::vector<double> same(E, 1000.0);
            const int64_t lanes = dom_lanes_rule(same.data(), E, sms), subs = 4 * sms;
            const int64_t warps = (lanes + DOM_GROUPS - 1) / DOM_GROUPS +
                                  (E - lanes + DOM_THREADS - 1) / DOM_THREADS;
            CHECK(lanes >= 0 && lanes <= E);
            if (E <= subs * DOM_THREADS) CHECK(warps <= subs + 2);
            if (E <= subs * DOM_GROUPS) CHECK(lanes == E);
            if (E > subs * DOM_THREADS) CHECK(lanes == 0);
        }
    std::vector<double> one(65536, 1.0);
    one[0] = 1e6;
    CHECK(dom_lanes_rule(one.data(), 65536, 152) == 1);
}

int main()
{
    adjoint();
    tensor_core_members();
    two_state_lanes();
    std::puts("rules ok");
    return 0;
}
