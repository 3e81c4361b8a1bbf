"""A body that fills the GPU and whose grid outgrows the cell arrays a handle
starts with: the many blocks of the launch that finds them too small stop
together, over and over, beside another handle, and what the step run again
with grown arrays builds is the oracle's."""
import numpy as np
import pytest

from mcmtop_b200 import _abi
from mcmtop_b200.deck import taylor_bar
from mcmtop_b200.solver import Solver
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


def test_many_blocks_stop_together():
    deck = taylor_bar(dx=0.14e-3)
    x = deck.x.copy()
    upper = x[:, 2] > 0.5 * (x[:, 2].min() + x[:, 2].max())
    x[upper, 2] += 400 * 2.0 * deck.materials[0].h
    deck = deck.replace(x=x)
    orc = Oracle(deck, openmp=True)
    counts = orc.get_int("nnbr")
    gl = orc.grid()[0]
    assert deck.np > 300000 and int(np.prod(gl.astype(np.int64))) > 65536
    bystander = Solver(taylor_bar(dx=0.8e-3), _abi.PREC_FP64_EXACT)
    before = bystander.download(["x", "v", "rho", "mass", "h"])
    for precision in (_abi.PREC_FP64_EXACT, _abi.PREC_FP64, _abi.PREC_MIXED):
        later = []
        for _ in range(4):
            sol = Solver(deck, precision)
            assert np.array_equal(sol.grid()[0], gl)
            assert np.array_equal(sol.neighbours()[0], counts)
            # cell counts that the stopped build had left would show in the next lists
            assert sol.run(2) == 2
            later.append(sol.neighbours()[0])
            sol.close()
        assert all(np.array_equal(later[0], nn) for nn in later[1:])
    after = bystander.download(["x", "v", "rho", "mass", "h"])
    for f in before:
        assert np.array_equal(before[f], after[f]), f
