"""The neighbour search's forms against each other and the oracle, entry for
entry: eight lanes per particle (small bodies, search_kind 2), four lanes
(from 24 000 particles) and one thread per particle (from 64 000), with one
smoothing length and with one per particle, several materials with kernel and
repulsive contact, the FP64 minimum distance wanted or not, and cells so full
that a row holds more candidates than the lanes' masks and a particle more
neighbours than its staging row."""
import dataclasses

import numpy as np
import pytest

from mcmtop_b200 import _abi
from mcmtop_b200.deck import taylor_bar, two_material_bar
from mcmtop_b200.solver import Solver
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


def wider(deck, factor):
    return deck.replace(materials=[dataclasses.replace(m, h=m.h * factor) for m in deck.materials])


def own_h(deck, seed=5):
    """A smoothing length per particle, between 0.8 and 1.1 of the material's."""
    rng = np.random.default_rng(seed)
    par = np.zeros((deck.np, 4))
    par[:, 1] = deck.materials[0].h * rng.uniform(0.8, 1.1, deck.np)
    return deck.replace(init_h_opt=1, pardata=par)


FORMS = {
    "plain": lambda dx: taylor_bar(dx=dx),
    "own_h": lambda dx: own_h(taylor_bar(dx=dx)),
    "kernel_contact": lambda dx: two_material_bar(dx=dx),
    "repulsive_contact": lambda dx: two_material_bar(dx=dx, contacttype=1),
    "full_cells": lambda dx: wider(taylor_bar(dx=dx), 1.7),
}


def lists(deck, kind, diagnostics, precision):
    s = Solver(deck, precision, nbr_stride=520)
    s.set_tuning(search_kind=kind)
    s.set_diagnostics(diagnostics)
    s.step_a()
    out = list(s.neighbours())
    if deck.contacttype > 0:
        out += list(s.contacts())
    if diagnostics:
        out.append(s.download(["mindist"])["mindist"])
    st = s.stats()
    s.close()
    return out + [np.array([st["max_nbr"]])]


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("diagnostics", [True, False])
@pytest.mark.parametrize("dx", [0.32e-3, 0.25e-3])   # 31 916: four lanes; 68 120: one thread
def test_forms_build_the_same_lists(form, diagnostics, dx):
    deck = FORMS[form](dx)
    a = lists(deck, 1, diagnostics, _abi.PREC_FP64_EXACT)
    b = lists(deck, 2, diagnostics, _abi.PREC_FP64_EXACT)
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("precision", [_abi.PREC_FP64_EXACT, _abi.PREC_MIXED])
def test_small_bodies_match_the_oracle(form, precision):
    deck = FORMS[form](0.8e-3) if form != "full_cells" else wider(taylor_bar(dx=0.8e-3), 2.4)
    sol, orc = Solver(deck, precision, nbr_stride=1000), Oracle(deck)
    sol.step_a()
    orc.step_a()
    nn, nbr, gn, _ = sol.neighbours()
    for i in range(deck.np):
        ref = orc.nbrlist(i + 1)
        assert np.array_equal(nbr[i, : nn[i]], ref), i
        assert gn[i] == len(orc.g_nbrlist(i + 1)), i
    g = sol.download(["mindist"])["mindist"]
    assert np.max(np.abs(g - orc.get("mindist"))) <= 1e-14 * np.max(np.abs(orc.get("mindist")))
