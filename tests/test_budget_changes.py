"""The budget of a binary64 step is that of the handle's grid and dt at the
time of the call, whether or not the step's cached face values were made for
them: rt_set_grid, or rt_set_dt with no valid coefficients, between a step
and its budget."""
import numpy as np
import pytest

from harness import configs

pytestmark = pytest.mark.gpu


def _grid(m, exp):
    d = [np.array(x, dtype=np.float64) for x in exp.d_interior]
    m.calc_grid([1.5 * x for x in d])
    from raytracer_3d_gb300 import _lib
    arrs = [np.ascontiguousarray(m.grid[ax]["dt"]) for ax in "xyzklm"]
    arrs += [np.ascontiguousarray(m.grid[ax]["t"]) for ax in "klm"]
    m._check(m._lib.rt_set_grid(m.handle, *[_lib.dptr(a) for a in arrs]), "rt_set_grid")


def _background_and_dt(m, exp):
    from raytracer_3d_gb300 import _lib
    m._check(m._lib.rt_set_background(m.handle, *[_lib.dptr(a) for a in (m.Nsqr, m.U, m.V)]), "rt_set_background")
    m.set_dt(0.5 * m.dt)


@pytest.mark.parametrize("change", [_grid, _background_and_dt])
@pytest.mark.parametrize("n", [(7, 3, 5, 2, 6, 4), (8, 8, 8, 6, 6, 8)])
def test_budget_after_a_change(n, change):
    import __graft_entry__ as g
    g.build()
    exp = configs.shear_mini(n=n)
    got = []
    for cached in (True, False):
        m = configs.build_model(exp, "fp64")
        m.integrate(3)
        if not cached:
            m.set_tuning("fast")      # the same states, but the face values make way for the fast step's
            m.set_dt(m.dt)
        change(m, exp)
        b, f = m.diagnose()
        got.append(([b[k] for k in sorted(b)], [f[k] for k in sorted(f)]))
        m.close()
    assert got[0][0] == got[1][0]
    assert all(np.array_equal(x, y) for x, y in zip(got[0][1], got[1][1]))
