"""Split steps on a handle whose fused run has ended (the caller goes on past the
end time of that run): they compute what they compute on another handle with the
same state."""
import numpy as np
import pytest

from mcmtop_b200 import _abi
from mcmtop_b200.deck import fluid_column, taylor_bar
from mcmtop_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [_abi.PREC_FP64_EXACT, _abi.PREC_FP64, _abi.PREC_MIXED])
@pytest.mark.parametrize("make", [lambda **kw: taylor_bar(dx=0.8e-3, **kw), lambda **kw: fluid_column(dx=50e-3, **kw)],
                         ids=["bar", "column"])
def test_steps_go_on(make, precision):
    a = Solver(make(endtime=1.0e-30), precision)
    assert a.run(5) < 5 and a.ended
    state = a.download()
    b = Solver(make(), precision)
    b.upload(state)
    b.dt, b.dtold = a.dt, a.dtold
    for s in (a, b):
        s.step_a()
        s.dt_update()
        s.step_b()
        s.step_c()
    got, want = a.download(["x", "v", "rho", "e", "sigma", "a"]), b.download(["x", "v", "rho", "e", "sigma", "a"])
    assert not np.array_equal(got["rho"], state["rho"])
    for f in want:
        assert np.array_equal(got[f], want[f]), f
    assert a.last_critts == b.last_critts
