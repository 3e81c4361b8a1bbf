"""A body in two parts far from one another: a grid of 55 000 cells, nearly all
empty.  The lists are the oracle's, and the cell list takes little longer than
that of the body in one piece (bound: three times; it was twelve when its
launches were sized by the particles alone)."""
import numpy as np
import pytest

from mcmtop_b200 import _abi
from mcmtop_b200.deck import taylor_bar
from mcmtop_b200.solver import Solver
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


def apart(deck, cells):
    x = deck.x.copy()
    upper = x[:, 2] > 0.5 * (x[:, 2].min() + x[:, 2].max())
    x[upper, 2] += cells * 2.0 * deck.materials[0].h
    return deck.replace(x=x)


@pytest.mark.parametrize("precision", [_abi.PREC_FP64_EXACT, _abi.PREC_FP64, _abi.PREC_MIXED])
def test_lists_in_a_sparse_grid(precision):
    deck = apart(taylor_bar(dx=0.8e-3), 6000)
    sol, orc = Solver(deck, precision), Oracle(deck)
    assert np.prod(orc.grid()[0].astype(np.int64)) > 50000
    for _ in range(2):
        assert sol.step() and orc.step()
    nn, nbr, _, _ = sol.neighbours()
    assert np.array_equal(sol.grid()[0], orc.grid()[0])
    for i in range(deck.np):
        assert np.array_equal(nbr[i, : nn[i]], orc.nbrlist(i + 1)), i


def test_time_of_the_cell_list():
    times = []
    for cells in (0, 6000):
        sol = Solver(apart(taylor_bar(dx=0.8e-3), cells), _abi.PREC_MIXED)
        sol.run(10)
        best = np.inf
        for _ in range(5):
            sol.profile(True)
            sol.run(20)
            best = min(best, sol.profile_report()["cell_list"][0])
            sol.profile(False)
        times.append(best)
        sol.close()
    assert times[1] <= 3.0 * times[0], times
