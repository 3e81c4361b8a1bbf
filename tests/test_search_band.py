"""The band within which the search's FP32 distances leave the decision to FP64,
against the rounding of those distances: x relative to the grid's origin, from
grids of a few cells to the longest that the grid check lets through."""
from host_program import run

PROGRAM = r"""
#include "common.cuh"
#include <cmath>
#include <cstdio>
#include <random>
int main() {
    std::mt19937_64 rng(1);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    for (double cells = 3.0; cells < 1.1e9; cells *= 2.3)
        for (double cell : {1.0, 0.0371, 1750.0}) {
            const int n = (int)cells;
            double worst = 0.0;
            for (int k = 0; k < 20000; ++k) {
                // a pair within reach of each other, anywhere in x, apart in one cell's y and z
                const double x = u(rng) * (n - 1) * cell, dx = (2.0 * u(rng) - 1.0) * cell;
                const double y = u(rng) * cell, dy = (2.0 * u(rng) - 1.0) * cell;
                const float fx = -(float)x - -(float)(x + dx), fy = -(float)y - -(float)(y + dy);
                const double d2 = dx * dx + dy * dy;
                worst = std::fmax(worst, std::fabs((double)std::fmaf(fx, fx, fy * fy) - d2));
            }
            std::printf("%d %.17g %.17g\n", n, worst, (double)mcm::search_band(n, (float)cell));
        }
}
"""


def test_band_covers_the_rounding(tmp_path):
    rows = [line.split() for line in run(str(tmp_path), PROGRAM).splitlines()]
    assert len(rows) > 60 and int(rows[-1][0]) > 4e8
    for n, worst, band in rows:
        # both decisions lean on it: reached by neither, and not far from what is needed
        assert float(worst) <= 0.5 * float(band), n
