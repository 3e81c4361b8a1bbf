"""A needle at the far end of a grid of more than 10^8 cells in x, where FP32
coordinates relative to the grid's origin lie many cells apart: the lists are
still the oracle's, entry for entry."""
import numpy as np
import pytest

from mcmtop_b200 import _abi
from mcmtop_b200.deck import fluid_column
from mcmtop_b200.solver import Solver
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


def needle(distance):
    d = fluid_column(dx=50e-3)
    dx = d.materials[0].h / 1.3
    rng = np.random.default_rng(3)
    i, j, k = np.meshgrid(np.arange(60), np.arange(2), np.arange(2), indexing="ij")
    x = np.stack([i.ravel(), j.ravel(), k.ravel()], axis=1) * dx
    x = x + rng.uniform(-0.1, 0.1, x.shape) * dx
    x = np.concatenate([x, x + [distance, 0.0, 0.0]])
    n = len(x)
    return d.replace(x=x, v=np.zeros_like(x), mat=np.ones(n, dtype=np.int32), dispbc=np.zeros(n, dtype=np.int32),
                     sym_flag=(0,) * 6, mirr_opt=0, base_a=(0.0, 0.0, 0.0))


@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("precision", [_abi.PREC_FP64_EXACT, _abi.PREC_MIXED])
def test_lists_match_the_oracle(precision, kind):
    # just past a power of two, where FP32 numbers are 256 length units apart
    deck = needle(2.0 ** 31 * 1.01)
    sol, orc = Solver(deck, precision), Oracle(deck)
    sol.set_tuning(search_kind=kind)
    gl = sol.grid()[0]
    assert np.array_equal(gl, orc.grid()[0]) and 1.0e8 < gl[0] < 2.0e8 and gl[1] == gl[2] == 1
    sol.step_a()
    orc.step_a()
    nn, nbr, _, _ = sol.neighbours()
    for i in range(deck.np):
        assert np.array_equal(nbr[i, : nn[i]], orc.nbrlist(i + 1)), i
    sol.close()
