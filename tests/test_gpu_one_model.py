"""The constitutive kernel of bodies with one model (9 or 10) against the one for
every model, which a body with a second, unused material of another model takes.
Bounds: the FP64-exact step has no contraction, so bitwise; the others' may
contract differently, which moves a step's result by some 2^-53 of a term (and,
through a neighbour's FP32 record, by 2^-24 of a pair's term), 100 terms that
exceed their sum by less than a thousand times."""
import numpy as np
import pytest

from mcmtop_b200 import _abi
from mcmtop_b200.deck import copper_model10, fluid_column, taylor_bar, water_model9
from mcmtop_b200.solver import Solver

pytestmark = pytest.mark.gpu

FIELDS = ["x", "v", "rho", "e", "p", "c", "efps", "sigma", "q"]
BOUND = {_abi.PREC_FP64_EXACT: 0.0, _abi.PREC_FP64: 1e5 * 2.0 ** -53, _abi.PREC_MIXED: 1e5 * 2.0 ** -24}


@pytest.mark.parametrize("diagnostics", [True, False])
@pytest.mark.parametrize("precision", BOUND)
@pytest.mark.parametrize("name", ["bar", "column"])
def test_one_model_as_all_models(name, precision, diagnostics):
    deck = taylor_bar(dx=0.8e-3) if name == "bar" else fluid_column(dx=40e-3)
    h = deck.materials[0].h
    other = water_model9(h) if name == "bar" else copper_model10(h)
    out = []
    for d in (deck, deck.replace(materials=list(deck.materials) + [other])):
        sol = Solver(d, precision)
        sol.set_diagnostics(diagnostics)
        assert sol.run(3) == 3
        out.append(sol.download(FIELDS))
        sol.close()
    for f in FIELDS:
        scale = float(np.max(np.abs(out[0][f])))
        assert np.max(np.abs(out[0][f] - out[1][f])) <= BOUND[precision] * scale, f
