// The std-dev heuristic's decision as the reference takes it, shared by the
// octree builds.
#pragma once

#include <cstdint>

#include "xn_bricks.h"

namespace xn {
namespace heur {

__device__ __forceinline__ uint64_t umin64(uint64_t a, uint64_t b) { return a < b ? a : b; }

__device__ __forceinline__ uint64_t clamped_count(const GridDev& g, uint64_t ox, uint64_t oy, uint64_t oz, uint64_t e) {
    return (umin64(g.dx, ox + e) - ox) * (umin64(g.dy, oy + e) - oy) * (umin64(g.dz, oz + e) - oz);
}

// Grid::stddev_scan (Grid.cpp:139-214) run literally, the sequential double
// loop in z, y, x order, over the cell's part of the grid.
static __device__ __noinline__ bool sequential_split(const GridDev& g, uint64_t x0, uint64_t y0, uint64_t z0, uint64_t e,
                                              const unsigned long long* s1, double threshold) {
    const uint64_t x1 = umin64(g.dx, x0 + e), y1 = umin64(g.dy, y0 + e), z1 = umin64(g.dz, z0 + e);
    const double nd = (double)((x1 - x0) * (y1 - y0) * (z1 - z0));
    double avg[4];
    for (int c = 0; c < 4; ++c) avg[c] = (double)s1[c] / nd;
    double s = 0.0;
    for (uint64_t z = z0; z < z1; ++z)
        for (uint64_t y = y0; y < y1; ++y)
            for (uint64_t x = x0; x < x1; ++x) {
                const uint32_t v = __ldg(g.vox + x + (uint64_t)g.dx * (y + (uint64_t)g.dy * z));
                const double d0 = (double)(v & 0xFFu) - avg[0];
                const double d1 = (double)((v >> 8) & 0xFFu) - avg[1];
                const double d2 = (double)((v >> 16) & 0xFFu) - avg[2];
                const double d3 = (double)(v >> 24) - avg[3];
                s += ((d0 * d0 + d1 * d1) + d2 * d2) + d3 * d3;
            }
    return sqrt(s / nd) > threshold;
}

// Cells of 2^k voxels a side up to this that lie inside the grid: there the
// reference's sum is exact in any order.  The mean is a multiple of 2^-3k, so
// the squares and their sums are multiples of 2^-6k, and with n = 2^3k voxels of
// four bytes the sum is below n 2^16: 9k + 16 bits, 52 for k = 4.  It is E / n,
// and the square root below is the reference's own.
constexpr uint64_t EXACT_CELL = 16;

// Whether the standard deviation sqrt(E)/n, E = n sum(x^2) - sum(x)^2 exact,
// is above the threshold, as the reference's sequential double sum decides:
// that sum differs from the exact value by at most (n + 16) 2^-52 relative,
// and inside that band its own loop decides (seq), but for cells of EXACT_CELL
// and below.
static __device__ __forceinline__ bool stddev_split(double E, uint64_t n, double threshold, bool& seq) {
    const double nd = (double)n;
    const double sd = sqrt(E / (nd * nd));
    const double band = (nd + 16.0) * 2.220446049250313e-16 * sd + 1e-300;
    seq = fabs(sd - threshold) <= band;
    return sd > threshold;
}

}  // namespace heur
}  // namespace xn
