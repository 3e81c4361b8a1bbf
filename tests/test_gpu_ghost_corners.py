"""Real particles beyond a plane, in cells that receive ghosts.  A cell that two
planes mirror into, or that holds reals and ghosts, is refused; a lone particle
beyond one plane is mirrored through the others as the oracle has it, also where
the cell between holds ghosts of the earlier of two planes only."""
import itertools

import numpy as np
import pytest

from mcmtop_b200 import _abi
from mcmtop_b200.deck import fluid_column
from mcmtop_b200.solver import Solver
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


def deck(cells, planes):
    """One particle at each position (in cells), walls at 0 on the axes of `planes`."""
    d = fluid_column(dx=50e-3)
    x = np.array(cells, dtype=np.float64) * 2.0 * d.materials[0].h
    n = len(x)
    return d.replace(x=x, v=np.zeros_like(x), mat=np.ones(n, dtype=np.int32), dispbc=np.zeros(n, dtype=np.int32),
                     sym_flag=tuple(f for p in planes for f in (p, 0)), base_a=(0.0, 0.0, 0.0))


FAR = (6.5, 6.5, 6.5)
REFUSED = {
    "two_planes_into_one_cell_xz": ([(0.5, 3.5, -0.3), (-0.3, 3.5, 0.5), FAR], (1, 0, 1)),
    "two_planes_into_one_cell_xy": ([(0.5, -0.3, 3.5), (-0.3, 0.5, 3.5), FAR], (1, 1, 0)),
    "two_planes_into_one_cell_yz": ([(3.5, 0.5, -0.3), (3.5, -0.3, 0.5), FAR], (0, 1, 1)),
    "a_real_below_its_mirror": ([(3.5, 3.5, 0.5), (3.5, 3.5, -0.3), FAR], (0, 0, 1)),
    "three_planes": ([(0.5, -0.3, 0.5), (-0.3, 0.5, 0.5), FAR], (1, 1, 1)),
}


@pytest.mark.parametrize("name", REFUSED)
def test_collisions_are_refused(name):
    with pytest.raises(_abi.MCMError) as e:
        Solver(deck(*REFUSED[name]), _abi.PREC_FP64_EXACT)
    assert e.value.code == _abi.MCM_EGHOST_LAYER


@pytest.mark.parametrize("at", [p for p in itertools.product((-0.3, 0.5, 2.5), repeat=3)])
def test_lone_particle_as_the_oracle(at):
    d = deck([at, FAR], (1, 1, 1))
    sol, orc = Solver(d, _abi.PREC_FP64_EXACT), Oracle(d)
    par, gx, gv = sol.ghosts()
    opar, ogx, ogv = orc.ghosts()
    assert np.array_equal(par, opar) and np.array_equal(gx, ogx) and np.array_equal(gv, ogv)
