"""The momentum gather's records, which the constitutive update writes: a second
momentum sum on the same state, whose records are formed from the stored state,
gives the same accelerations.  Ghosts of one plane and of several, periodic
images, the cap model's two triangles, particles outside the grid's cells, the
corrected form.  Bounds: the FP64-exact records are the same expressions without
contraction, so bitwise; the FP64-fast ones may differ by the contraction of
(sigma - q), and the FP32 ones by one rounding of a term: 2^-53 and 2^-24 of a
term, 100 terms that exceed their sum by less than a thousand times."""
import numpy as np
import pytest

from mcmtop_b200 import _abi
from mcmtop_b200.deck import MMMSG, fluid_column, periodic_layer, sand_model4, taylor_bar
from mcmtop_b200.solver import Solver

pytestmark = pytest.mark.gpu


def sand():
    return taylor_bar(dx=0.8e-3, velocity=60.0, material=sand_model4(0.0), units=MMMSG)


DECKS = {
    "bar": lambda: taylor_bar(dx=0.8e-3),
    "bar_corrected": lambda: taylor_bar(dx=0.8e-3, disctype=1),
    "column": lambda: fluid_column(dx=40e-3),
    "layer": lambda: periodic_layer(dx=40e-3),
    "sand": sand,
}
BOUND = {_abi.PREC_FP64_EXACT: 0.0, _abi.PREC_FP64: 1e5 * 2.0 ** -53, _abi.PREC_MIXED: 1e5 * 2.0 ** -24}


@pytest.mark.parametrize("precision", BOUND)
@pytest.mark.parametrize("name", DECKS)
def test_second_sum_on_the_same_state(name, precision):
    if name == "bar_corrected" and precision == _abi.PREC_MIXED:
        pytest.skip("the mixed step has the simple form only")
    sol = Solver(DECKS[name](), precision)
    for _ in range(2):
        assert sol.step()
    sol.step_a()
    sol.step_b()
    a = sol.download(["a"])["a"]
    sol.step_b()
    b = sol.download(["a"])["a"]
    assert np.max(np.abs(a)) > 0.0
    assert np.max(np.abs(a - b)) <= BOUND[precision] * np.max(np.abs(a))
