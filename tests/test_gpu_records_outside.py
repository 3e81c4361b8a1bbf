"""Particles outside the grid's cells (an uploaded box smaller than the body):
no neighbours, none of theirs, and the momentum records that the constitutive
update writes for all positions are those formed from the stored state.  Both
are made of the same FP64 values; where the compiler contracts (sigma - q) / rho^2
in one and not the other they differ by a rounding of a term, 2^-53 or (the
mixed records) 2^-24, and the terms of a sum add up to less than 100 times the
largest acceleration.

The one-model constitutive kernels against the one for every model, measured by
what the steps change: the same rounding per step, in three steps."""
import numpy as np
import pytest

from mcmtop_b200 import _abi
from mcmtop_b200.deck import copper_model10, fluid_column, periodic_layer, taylor_bar, water_model9
from mcmtop_b200.solver import Solver

pytestmark = pytest.mark.gpu

EPS = {_abi.PREC_FP64_EXACT: 0.0, _abi.PREC_FP64: 2.0 ** -53, _abi.PREC_MIXED: 2.0 ** -24}
DECKS = {
    "bar": (lambda: taylor_bar(dx=0.8e-3), 2),
    "bar_corrected": (lambda: taylor_bar(dx=0.8e-3, disctype=1), 2),
    "column": (lambda: fluid_column(dx=40e-3), 2),
    "layer": (lambda: periodic_layer(dx=40e-3), 2),
}


@pytest.mark.parametrize("precision", EPS)
@pytest.mark.parametrize("name", DECKS)
def test_records_with_particles_outside(name, precision):
    make, axis = DECKS[name]
    if name == "bar_corrected" and precision == _abi.PREC_MIXED:
        pytest.skip("the mixed step has the simple form only")
    sol = Solver(make(), precision)
    assert sol.step()
    state = sol.download()
    x = state["x"]
    box = np.stack([x.min(axis=0), x.max(axis=0)], axis=1)
    box[axis, 1] = box[axis, 0] + 0.6 * (box[axis, 1] - box[axis, 0])
    sol.upload(state, bbox=box.ravel())
    sol.step_a()
    sol.step_b()
    a = sol.download(["a"])["a"]
    gl, lo, size = sol.grid()
    outside = size[axis] * (x[:, axis] - lo[axis]) > gl[axis] + 1e-6
    assert 0.1 < np.mean(outside) < 0.5
    nn, nbr, _, _ = sol.neighbours()
    own = 1 if name == "bar_corrected" else 0
    assert np.all(nn[outside] == own) and np.all(nn[~outside] > own)
    ids = np.flatnonzero(outside) + 1
    inside = nbr[~outside]
    assert not np.isin(inside[np.arange(inside.shape[1]) < nn[~outside, None]], ids).any()
    sol.step_b()
    b = sol.download(["a"])["a"]
    assert np.max(np.abs(a)) > 0.0
    assert np.max(np.abs(a - b)) <= 100 * EPS[precision] * np.max(np.abs(a))


@pytest.mark.parametrize("precision", EPS)
@pytest.mark.parametrize("name", ["bar", "column"])
def test_one_model_changes_what_all_models_change(name, precision):
    deck = DECKS[name][0]()
    h = deck.materials[0].h
    other = water_model9(h) if name == "bar" else copper_model10(h)
    out = []
    for d in (deck, deck.replace(materials=list(deck.materials) + [other])):
        sol = Solver(d, precision)
        start = sol.download(["x", "v"])
        assert sol.run(3) == 3
        end = sol.download(["x", "v"])
        out.append({f: end[f] - start[f] for f in end})
        sol.close()
    # a difference of two positions is known to a rounding of the positions
    floor = {f: 4 * 2.0 ** -53 * np.max(np.abs(v)) for f, v in end.items()}
    for f in out[0]:
        bound = 3 * 100 * EPS[precision] * np.max(np.abs(out[0][f])) + (floor[f] if EPS[precision] else 0.0)
        assert np.max(np.abs(out[0][f] - out[1][f])) <= bound, f
