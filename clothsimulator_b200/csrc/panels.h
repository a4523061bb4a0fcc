// Host side of the on-chip solvers' shared-memory budget (resident.cu, group.cu).
#pragma once
#include <algorithm>

// How many of the block slots of each of a CTA's `n` slices (`width` slots, one panel each) it keeps in
// shared memory when that holds `cap` panels; a slice's other slots are read from L2.  What exceeds
// the budget is dealt evenly over the slices, since the slowest warp sets an iteration's time; a slice
// narrower than its share leaves the rest to the next ones, and what the last slices were too narrow
// for is taken from the earlier ones, a panel each in turn.  The kept panels sum to
// min(cap, sum of width): the kernels lay them out one after another without a further check.
inline void keptPanels(const int* width, int n, int cap, int* keep) {
    int panels = 0;
    for (int j = 0; j < n; j++) panels += width[j];
    const int over = std::max(panels - std::max(cap, 0), 0);
    int out = 0;
    for (int j = 0; j < n; j++) {
        const int o = std::min(width[j], (int)((long long)over * (j + 1) / n) - out);
        keep[j] = width[j] - o;
        out += o;
    }
    while (out < over)
        for (int j = n - 1; j >= 0 && out < over; j--)
            if (keep[j] > 0) {
                keep[j]--;
                out++;
            }
}
