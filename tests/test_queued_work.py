"""Set-up calls right behind queued steps: the steps still see the tables they
were queued with, and the next ones the new ones."""
import numpy as np
import pytest

from harness import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision, variant", [("fp32", "tma"), ("fp64", "split"), ("fp64", "fast")])
@pytest.mark.parametrize("what", ["dt", "grid"])
def test_changes_do_not_reach_queued_steps(precision, variant, what):
    import __graft_entry__ as g
    g.build()
    n = (32, 32, 16, 8, 8, 8)
    exp = configs.shear_mini(n=n)
    steps = 60                      # tens of milliseconds on the GPU
    got = []
    for wait in (True, False):
        m = configs.build_model(exp, precision, padded=False)
        m.set_tuning(variant, 8, 256)
        m.set_state()
        m.integrate(steps)
        if wait:
            m.sync()
        if what == "dt":
            m.set_dt(0.5 * m.dt)
        else:
            m.calc_grid([1.25 * np.array(x, dtype=np.float64) for x in exp.d_interior])
            m.calc_parameter()
        m.integrate(3)
        got.append(m.get_state())
        m.close()
    assert np.isfinite(got[0]).all()
    assert np.array_equal(got[0], got[1])
