// rules.hpp -- host-side choices that depend on sizes alone.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace magpy {

// What the adjoint keeps for the sweep back beside a segment's moments (3 planes of
// one float a particle and step): the dipolar fields of a step's two stages, 6
// planes more, of every step of the run (which then needs no checkpoints), of the
// segment being swept, or of none.  The kept planes are bounded by 4 GiB, and by
// a sixteenth of the memory that is free, so that objects made side by side never
// take most of it from the plans that follow them.  Up to 64 MiB are kept without
// asking what is free (the answer takes 60 us, a seventh of a small gradient).
enum class AdjointKeep { none, segment, whole };
constexpr size_t ADJOINT_KEEP_UNASKED = (size_t)64 << 20;

inline AdjointKeep adjoint_keep(size_t steps, size_t every, size_t particles, size_t free_bytes)
{
    const size_t limit = std::max(ADJOINT_KEEP_UNASKED, std::min((size_t)4 << 30, free_bytes / 16));
    const auto fits = [&](size_t n) {
        return particles == 0 || n <= limit / 9 / sizeof(float) / particles;
    };
    if (fits(steps)) return AdjointKeep::whole;
    return fits(std::min(steps, every)) ? AdjointKeep::segment : AdjointKeep::none;
}

// Members per CTA of the single-CTA tensor-core kernel, one CTA an SM: the fewest
// that need no more waves of CTAs than 32 (a CTA's step takes less time with fewer:
// 3.75, 3.9, 4.2 and 4.9 us with 8, 16, 20 and 32 members of 64 particles, 2.63 and
// 2.65 with 8 and 32 of 16).
inline int tc_members(int64_t E, int sms)
{
    const int64_t waves = ((E + 31) / 32 + sms - 1) / sms;
    int nm = 32;
    while (nm > 8 && (E + nm - 5) / (nm - 4) <= waves * sms) nm -= 4;
    return nm;
}

// Two-state kernel: particles per warp, with one lane each and with five.
constexpr int DOM_THREADS = 32, DOM_GROUPS = 6;

// How many of E particles, in descending order of their expected relative step
// counts, get five lanes.  Five lanes take a particle through a step in 0.42 of the
// time and in 2.4 times the FP64 issue of one thread.  The first ones of the order
// get them while every warp still has a sub-partition of its own; past that, those
// that would need more than half the time of the whole batch by themselves.
inline int64_t dom_lanes_rule(const double *steps, int64_t E, int sms)
{
    const int64_t subs = 4 * (int64_t)sms;
    const int64_t fill = (subs * DOM_THREADS - E) * DOM_GROUPS / (DOM_THREADS - DOM_GROUPS);
    int64_t lanes = std::min(E, std::max<int64_t>(0, fill));
    double sum = 0.0;
    for (int64_t e = 0; e < E; e++) sum += steps[e];
    const double alone = std::max(1.3 * sum / (double)E, 0.5 * sum / (double)(subs * DOM_THREADS));
    while (lanes < E && steps[lanes] > alone) lanes++;
    return lanes;
}

}  // namespace magpy
