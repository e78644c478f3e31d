// How many steps one launch may advance an instance by (see Span in
// asg_engine.cuh), as far as its spike list can hold them.  Host arithmetic on
// the descriptor's sizes alone.
#pragma once

#include <algorithm>
#include <cstdint>

namespace asg {

// Most steps of a window of `steps` in which one cell spikes: a spike in a
// substep keeps the cell refractory for `ref_steps` substeps, and a step lists
// the cell once.
inline std::int64_t most_spikes(int steps, int substeps, int ref_steps) {
    const std::int64_t apart = static_cast<std::int64_t>(std::max(ref_steps, 0)) + 1;
    const std::int64_t spikes = (static_cast<std::int64_t>(steps) * substeps + apart - 1) / apart;
    return std::min<std::int64_t>(steps, spikes);
}

// The largest L <= want whose launches' spikes fit a spike list whatever the
// cells do: its header counts records in `count_bits`, and a record's edge offset
// and the push's index over the launch's edges (which overshoots by up to four
// strides of 128 threads x (2^16 + 2 per SM) blocks, below 2^26) have 32.  A
// cell with a refractory time of L steps or more counts once, as in a launch
// of one step; without one, five steps fit 845 million edges.  1 (a launch per
// step) where nothing more fits.
inline int span_that_fits(int want, std::uint64_t neurons, std::uint64_t edges, int substeps,
                          int ref_steps, int count_bits) {
    for (int L = want; L > 1; --L) {
        const auto s = static_cast<std::uint64_t>(most_spikes(L, substeps, ref_steps));
        if (s * neurons < (1ull << count_bits) && s * edges <= (1ull << 32) - (1ull << 26)) return L;
    }
    return 1;
}

}  // namespace asg
