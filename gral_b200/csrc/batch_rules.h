// batch_rules.h -- the layout a batch runs in, and how its situations are split into the sets that the row
// chains run one after the other (host code without CUDA, also compiled by the CPU tests).
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

// Whether a batch runs faster in the interleaved layout; levels: those swept in a column.  A batched sweep
// waits for its wavefront (rows + columns steps) and works through its groups of 32 (per column and group), both level
// by level; the row chains take a time per column and situation that depends on the levels only by
// their coefficients and records, and a small one per row and column.  ms of an iteration, fitted
// to 276 pairs of 48x48 .. 400x400 grids, 32 to 256 situations and 8 to 44 levels (a pick costs 0.3 % on average, 16 %
// at most; without the levels it cost up to 59 %).  Row chains / interleaved, 64 situations of 200x200: 8 levels, model 1
// 14.9 / 11.5; 28 levels 21.0 / 21.0; 44 levels 26.2 / 29.0, model 0 29.9 / 36.1, model 2 52.5 / 58.7.
inline bool interleaved_pays(int n, int nii, int njj, int levels, int model) {
    if (n < 32) return false;
    static const double P[3][3] = {{6.57e-6, 1.01e-7, 2.7e-3}, {4.16e-6, 1.33e-7, 1.7e-3}, {9.28e-6, 2.42e-7, 3.5e-3}};
    static const double I[3][4] = {{13.4e-3, 1.27e-3, 4.3e-6, 2.24e-6}, {14.5e-3, 0.884e-3, 17.9e-6, 1.78e-6}, {20.8e-3, 2.14e-3, 19.3e-6, 3.46e-6}};
    const double cols = (double)nii * njj, groups = (n + 31) / 32, steps = nii + njj;
    const double *p = P[model], *q = I[model];
    return n * cols * (p[0] + p[1] * levels) + steps * p[2] > steps * (q[0] + q[1] * levels) + groups * cols * (q[2] + q[3] * levels);
}

}  // namespace gral
