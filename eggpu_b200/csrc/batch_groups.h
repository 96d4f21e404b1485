// Chooses how many panels of a batch are solved together (host code without CUDA, so that
// it can be checked without a GPU).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

namespace egpr {

// Sweeps that a column is expected to take: the stop rule's residual starts below 2 and fell
// to 0.34-0.43 of it per sweep on R-MAT and uniform graphs (alpha 0.85; alpha is the bound,
// which only a chain comes near to).
inline int32_t expected_sweeps(double alpha, double tol, int32_t max_iter, int32_t n) {
    if (!(tol > 0.0) || !(alpha > 0.0 && alpha < 1.0)) return max_iter;
    const double bound = std::ceil(std::log(0.5 * tol * (double)n) / std::log(0.5 * alpha));
    return (int32_t)std::min((double)max_iter, std::max(1.0, bound));
}

// Panels (of 32 columns) per group.  The results of a group travel to the host while the
// next one is solved, so small groups hide more of the read-back, and large ones lose less
// at the ends of the launches.  Times in ms, fitted on B200 (R-MAT scale 18 to 22, uniform
// graphs, 8 to 65 M entries, 10 to 200 sweeps, 64 to 256 columns): a sweep of p panels
// takes p * 22 ps per entry + 0.15 ms, set-up and the FP64 pass two sweeps more, a panel's
// results 256 bytes per vertex at 55 GB/s.  Over the 62 batches of the fit the choice took
// 0.3% longer than the best of 1, 2, 3, 4, 6 and 8 panels, 5.5% at most, and was never slower
// than one group; three panels always were up to 18% slower than one group (R-MAT scale
// 18, 40 entries per vertex, 256 columns, 200 sweeps: 341 ms, 289 in one group).
inline int32_t batch_group_panels(int64_t entries, int32_t n, int32_t panels, int32_t sweeps, int32_t most) {
    const double panel = 22e-9 * (double)entries, launch = 0.15, copy = (double)n * 256.0 / 55e6;
    int32_t best = most;
    double best_ms = INFINITY;
    for (int32_t g = std::min(panels, most); g >= 1; --g) {
        double solved = 0.0, copied[2] = {0.0, 0.0};  // when the last solve and the last two copies end
        for (int32_t left = panels; left > 0; left -= g) {
            const int32_t p = std::min(g, left);
            solved = std::max(solved, copied[0]) + (sweeps + 2.0) * (p * panel + launch);  // two result buffers
            copied[0] = copied[1];
            copied[1] = std::max(solved, copied[1]) + p * copy;
        }
        if (copied[1] < best_ms) {
            best_ms = copied[1];
            best = g;
        }
    }
    return best;
}

}  // namespace egpr
