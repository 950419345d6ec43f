// unit_sets.h -- how a batch's situations are split into the sets that the row chains run one after the
// other (host code without CUDA, also compiled by the CPU tests).
#pragma once

#include <algorithm>
#include <cstddef>

namespace gral {

constexpr int kCounterSlots = 64;   // launches per phase with task counters of their own

// the smallest set: every set takes a counter slot, and there are kCounterSlots of them
inline int min_units(int nb) { return std::max(1, (nb + kCounterSlots - 1) / kCounterSlots); }

// sets of equal size with at most `fit` situations, but no smaller than min_units
inline int set_units(int nb, size_t fit) {
    const int units = std::max(min_units(nb), (int)std::min<size_t>((size_t)nb, std::max<size_t>(fit, 1)));
    const int sets = (nb + units - 1) / units;
    return (nb + sets - 1) / sets;
}

// the next smaller set to try when there is no memory for one of `units`; 0 when there is none
inline int fewer_units(int nb, int units) {
    if (units <= min_units(nb)) return 0;
    return std::max(min_units(nb), std::min(units - 1, set_units(nb, (size_t)(units + 1) / 2)));
}

}  // namespace gral
