"""Boxes that give no usable grid: a body whose positions are not numbers and one
strewn over more cells than can be counted are refused; a body wholly beyond a
plane has no cells, so its particles have no neighbours and no ghosts and fly on
freely until the plane reflects them."""
import numpy as np
import pytest

from mcmtop_b200 import _abi
from mcmtop_b200.deck import fluid_column, taylor_bar
from mcmtop_b200.solver import Solver

pytestmark = pytest.mark.gpu

PRECISIONS = [_abi.PREC_FP64_EXACT, _abi.PREC_FP64, _abi.PREC_MIXED]


@pytest.mark.parametrize("precision", PRECISIONS)
def test_positions_that_are_not_numbers(precision):
    sol = Solver(taylor_bar(dx=0.8e-3), precision)
    state = sol.download()
    good = {f: a.copy() for f, a in state.items()}
    state["x"] = np.full_like(state["x"], np.nan)
    sol.upload(state)
    with pytest.raises(_abi.MCMError) as e:
        sol.step_a()
    assert e.value.code == _abi.MCM_EGRID_TOO_LARGE
    # the handle goes on with a state that has positions
    ref = Solver(taylor_bar(dx=0.8e-3), precision)
    lo, hi = good["x"].min(axis=0), good["x"].max(axis=0)
    sol.upload(good, bbox=np.stack([lo, hi], axis=1).ravel())
    assert sol.step() and ref.step()
    a, b = sol.download(["x", "v", "rho", "e"]), ref.download(["x", "v", "rho", "e"])
    assert all(np.array_equal(a[f], b[f]) for f in a)


@pytest.mark.parametrize("cells", [3.0e6, 4.0e8])
def test_more_cells_than_can_be_counted(cells):
    deck = taylor_bar(dx=0.8e-3)
    x = deck.x.copy()
    x[0] += cells * 2.0 * deck.materials[0].h
    with pytest.raises(_abi.MCMError) as e:
        Solver(deck.replace(x=x, sym_flag=(0,) * 6, mirr_opt=0), _abi.PREC_FP64_EXACT)
    assert e.value.code == _abi.MCM_EGRID_TOO_LARGE


@pytest.mark.parametrize("kind", [1, 2, 3])
@pytest.mark.parametrize("cells", [1.25, 2.25, 5.25, 40.25])
@pytest.mark.parametrize("precision", PRECISIONS)
def test_body_beyond_a_plane(precision, cells, kind):
    d = fluid_column(dx=50e-3)
    cell = 2.0 * d.materials[0].h
    x = d.x.copy()
    x[:, 0] -= x[:, 0].max() + cells * cell   # the nearest particle `cells` cells beyond the plane at x = 0
    v = np.tile([0.0, 0.01, 0.0], (d.np, 1))
    d = d.replace(x=x, v=v, sym_flag=(1, 0, 0, 0, 0, 0), base_a=(0.0, 0.0, 0.0))
    sol = Solver(d, precision)
    sol.set_tuning(search_kind=kind)
    gl = sol.grid()[0]
    assert gl[0] < 2
    nn, _, gn, _ = sol.neighbours()
    assert not gn.any() and len(sol.ghosts()[0]) == 0
    if gl[0] < 1:
        assert not nn.any()
    assert sol.step()
    got = sol.download(["x", "v"])
    if gl[0] < 1:
        xn = x + v * sol.dt
        xn[:, 0] = -xn[:, 0]
        assert np.max(np.abs(got["x"] - xn)) <= 1e-12 * np.max(np.abs(x))
    # the box of the first move is the one before the reflection; then an ordinary grid
    assert sol.step() and sol.step() and sol.grid()[0][0] >= 2
