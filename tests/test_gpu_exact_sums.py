"""The FP64-exact step's in-order sums on both sides of the size where a particle
has eight lanes (below 36 000) or one thread, against the CPU oracle: simple
and corrected SPH, ghost walls, contacts, a smoothing length per particle (the
divisions that the shared reciprocals do not cover), and a lattice without
jitter (differences and quotients that are exactly zero).  Bound: the
FP64-exact step's, 1e-13 of each field's range per step."""
import numpy as np
import pytest

from mcmtop_b200 import _abi
from mcmtop_b200.deck import fluid_column, taylor_bar, two_material_bar
from mcmtop_b200.solver import Solver
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


def own_h(deck, seed=5):
    rng = np.random.default_rng(seed)
    par = np.zeros((deck.np, 4))
    par[:, 1] = deck.materials[0].h * rng.uniform(0.8, 1.1, deck.np)
    return deck.replace(init_h_opt=1, pardata=par)


DECKS = {
    "bar": lambda s: taylor_bar(dx=(0.8e-3, 0.3e-3)[s]),
    "bar_corrected": lambda s: taylor_bar(dx=(0.8e-3, 0.3e-3)[s], disctype=1),
    "bar_own_h": lambda s: own_h(taylor_bar(dx=(0.8e-3, 0.3e-3)[s])),
    "bar_own_h_corrected": lambda s: own_h(taylor_bar(dx=(0.8e-3, 0.3e-3)[s], disctype=1)),
    "lattice": lambda s: taylor_bar(dx=(0.8e-3, 0.3e-3)[s], jitter=0.0),
    "column": lambda s: fluid_column(dx=(40e-3, 14.7e-3)[s]),
    "column_corrected": lambda s: fluid_column(dx=(40e-3, 14.7e-3)[s]).replace(disctype=1),
    "contact": lambda s: two_material_bar(dx=(0.8e-3, 0.3e-3)[s], contacttype=1),
    "contact_corrected": lambda s: two_material_bar(dx=(0.8e-3, 0.3e-3)[s], contacttype=1, disctype=1),
}


@pytest.mark.parametrize("size", [0, 1])
@pytest.mark.parametrize("name", DECKS)
def test_sums_match_oracle(name, size):
    deck = DECKS[name](size)
    assert (deck.np >= 36000) == bool(size)
    sol, orc = Solver(deck, _abi.PREC_FP64_EXACT), Oracle(deck, openmp=True)
    for _ in range(2):
        assert sol.step() and orc.step()
    g = sol.download(["x", "v", "a", "rho", "e", "p", "sigma", "rod", "spin"])
    for f in g:
        ref = np.asarray(orc.get(f))
        scale = float(np.max(np.abs(ref)))
        assert np.max(np.abs(g[f] - ref)) <= 2e-13 * scale if scale > 0 else not np.any(g[f]), f
    e = orc.energies()
    assert np.max(np.abs(sol.energies_now() - e)) <= 1e-12 * np.max(np.abs(e))
