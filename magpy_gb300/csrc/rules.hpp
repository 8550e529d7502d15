// rules.hpp -- host-side choices that depend on sizes alone.
#pragma once
#include <algorithm>
#include <cstddef>

namespace magpy {

// What the adjoint keeps for the sweep back beside a segment's moments (3 planes of
// one float a particle and step): the dipolar fields of a step's two stages, 6
// planes more, of every step of the run (which then needs no checkpoints), of the
// segment being swept, or of none.  The kept planes are bounded by 4 GiB, and by
// a sixteenth of the memory that is free, so that objects made side by side never
// take most of it from the plans that follow them.
enum class AdjointKeep { none, segment, whole };

inline AdjointKeep adjoint_keep(size_t steps, size_t every, size_t particles, size_t free_bytes)
{
    const size_t limit = std::min((size_t)4 << 30, free_bytes / 16);
    const auto fits = [&](size_t n) {
        return particles == 0 || n <= limit / 9 / sizeof(float) / particles;
    };
    if (fits(steps)) return AdjointKeep::whole;
    return fits(std::min(steps, every)) ? AdjointKeep::segment : AdjointKeep::none;
}

}  // namespace magpy
