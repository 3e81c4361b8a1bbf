"""Counts of cells and of the planes' layer cells at the largest grids that the
grid check lets through (2^31 - 1 cells): the chunks of the scans and the layers'
sequence do not wrap, and no loop over the cells has a signed 32-bit counter,
which would pass the last cell and turn negative."""
import os
import re

from host_program import run
from mcmtop_b200.build import CSRC

PROGRAM = r"""
#include "common.cuh"
#include <cstdio>
int main() {
    for (unsigned n : {0u, 1u, 4096u, 4097u, 2147479552u, 2147479553u, 2147483647u, 4294967294u})
        std::printf("%u ", (unsigned)mcm::scan_chunks(n));
    const int grids[4][3] = {{9, 8, 7}, {230000000, 3, 3}, {3, 230000000, 3}, {2, 2, 500000000}};
    for (const int *g : grids)
        for (unsigned active : {0u, 0x3fu, 0x15u}) {
            unsigned first[7];
            mcm::layer_starts(g, active, first);
            std::printf("%u %u ", (unsigned)first[5], (unsigned)first[6]);
        }
}
"""


def test_counts_do_not_wrap(tmp_path):
    got = [int(v) for v in run(str(tmp_path), PROGRAM).split()]
    want = [-(-n // 4096) for n in (0, 1, 4096, 4097, 2147479552, 2147479553, 2147483647, 4294967294)]
    for g in ((9, 8, 7), (230000000, 3, 3), (3, 230000000, 3), (2, 2, 500000000)):
        for active in (0, 0x3F, 0x15):
            area = [g[1] * g[2], g[1] * g[2], g[0] * g[2], g[0] * g[2], g[0] * g[1], g[0] * g[1]]
            area = [v if active >> p & 1 else 0 for p, v in enumerate(area)]
            want += [sum(area[:5]), sum(area)]
    assert got == want


def test_no_signed_counter_over_the_cells():
    with open(os.path.join(CSRC, "cells.cu")) as f:
        text = f.read()
    loops = re.findall(r"for \((\w+(?: \w+)*) (\w+) = [^;]*; \2 <=? ([^;]*);", text)
    over_cells = [(kind, bound) for kind, _, bound in loops if "ncells" in bound or bound == "T"]
    assert len(over_cells) >= 4
    assert all(kind in ("unsigned", "long long") for kind, _ in over_cells), over_cells
