"""Bodies whose linked-list grid outgrows the cell arrays a handle starts with
(65 536 cells): the step that finds them too small must touch nothing, and the
step run again with grown arrays (whose length is no multiple of the scan's
chunk) must give the reference's grid and neighbour sets."""
import numpy as np
import pytest

from mcmtop_b200 import _abi
from mcmtop_b200.deck import taylor_bar
from mcmtop_b200.solver import Solver
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


def split_bar(gap_cells):
    """A small bar whose upper half is moved up by gap_cells cells."""
    d = taylor_bar(dx=0.8e-3, length=8.0e-3)
    x = d.x.copy()
    upper = x[:, 2] > 0.5 * (x[:, 2].min() + x[:, 2].max())
    x[upper, 2] += gap_cells * 2.0 * d.materials[0].h
    return d.replace(x=x)


@pytest.mark.parametrize("precision", [_abi.PREC_FP64_EXACT, _abi.PREC_MIXED])
@pytest.mark.parametrize("gap", [8000, 25000])
def test_grid_grows(precision, gap):
    deck = split_bar(gap)
    bystander = Solver(taylor_bar(dx=0.8e-3), _abi.PREC_FP64_EXACT)
    before = bystander.download(["x", "v", "rho", "mass", "h"])
    sol, orc = Solver(deck, precision), Oracle(deck)
    for _ in range(2):
        assert sol.step() and orc.step()
    gl = sol.grid()[0]
    assert np.array_equal(gl, orc.grid()[0]) and int(np.prod(gl.astype(np.int64))) > 65536
    nn, nbr, _, _ = sol.neighbours()
    for i in range(deck.np):
        assert np.array_equal(np.sort(nbr[i, : nn[i]]), np.sort(orc.nbrlist(i + 1))), i
    after = bystander.download(["x", "v", "rho", "mass", "h"])
    for f in before:
        assert np.array_equal(before[f], after[f]), f
