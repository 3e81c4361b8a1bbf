"""Corrected SPH (disctype 1) with the FP64-fast gathers against the CPU oracle:
each of a particle's lanes forms the acceleration from the complete sums, so
it must not be added over the lanes again.  Bound: the FP64-fast step's
(1e-9 of each field's range)."""
import numpy as np
import pytest

from mcmtop_b200 import _abi
from mcmtop_b200.deck import fluid_column, taylor_bar
from mcmtop_b200.solver import Solver
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [lambda: taylor_bar(dx=0.8e-3, disctype=1),
                                  lambda: fluid_column(dx=50e-3).replace(disctype=1)],
                         ids=["bar", "column"])
@pytest.mark.parametrize("steps", [1, 8])
def test_corrected_fp64_matches_oracle(make, steps):
    deck = make()
    sol, orc = Solver(deck, _abi.PREC_FP64), Oracle(deck)
    for _ in range(steps):
        assert sol.step() and orc.step()
    g = sol.download(["x", "v", "a", "rho", "sigma"])
    for f in g:
        ref = np.asarray(orc.get(f))
        assert np.max(np.abs(g[f] - ref)) <= 1e-9 * max(np.max(np.abs(ref)), 1e-300), f
