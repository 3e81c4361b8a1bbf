"""A state uploaded without its box to a handle whose last call failed or ended
the run: the box is formed from the new positions, not left as it was."""
import numpy as np
import pytest

from mcmtop_b200 import _abi
from mcmtop_b200.deck import taylor_bar
from mcmtop_b200.solver import Solver

pytestmark = pytest.mark.gpu

PRECISIONS = [_abi.PREC_FP64_EXACT, _abi.PREC_FP64, _abi.PREC_MIXED]


def deck(**kw):
    return taylor_bar(dx=0.8e-3).replace(sym_flag=(0,) * 6, mirr_opt=0, **kw)


def moved(state, by):
    out = {f: a.copy() for f, a in state.items()}
    out["x"] = out["x"] + by
    return out


@pytest.mark.parametrize("precision", PRECISIONS)
def test_after_an_error(precision):
    sol = Solver(deck(), precision)
    state = sol.download()
    counts = sol.neighbours()[0]
    bad = moved(state, 0.0)
    bad["x"][0] = 1.0e30
    sol.upload(bad)
    with pytest.raises(_abi.MCMError):
        sol.step_a()
    sol.upload(moved(state, 256.0))   # (a power of two: few last bits move)
    sol.step_a()
    lo = sol.grid()[1]
    assert np.all(np.abs(lo - (256.0 + state["x"].min(axis=0))) < 0.1 * state["h"].max())
    assert np.mean(sol.neighbours()[0] == counts) > 0.99


@pytest.mark.parametrize("precision", PRECISIONS)
def test_after_the_end_of_a_run(precision):
    sol = Solver(deck(endtime=1.0e-30), precision)
    state = sol.download()
    counts = sol.neighbours()[0]
    assert sol.run(5) < 5 and sol.ended
    sol.upload(moved(state, 256.0))
    sol.step_a()
    lo = sol.grid()[1]
    assert np.all(np.abs(lo - (256.0 + state["x"].min(axis=0))) < 0.1 * state["h"].max())
    assert np.mean(sol.neighbours()[0] == counts) > 0.99
