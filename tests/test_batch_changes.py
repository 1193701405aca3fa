"""A batch follows what changes in its members between two calls: each gives
the result it gets alone."""
import numpy as np
import pytest

from harness import configs, interior

pytestmark = pytest.mark.gpu


def _set_dt(m, exp):
    m.set_dt(0.5 * m.dt)


def _new_grid(m, exp):
    """another z spacing: the bottom cell's height enters the forcing"""
    d = [np.array(x, dtype=np.float64) for x in exp.d_interior]
    d[2] = d[2] * 1.25
    m.calc_grid(d)
    m.calc_parameter()


CHANGES = {"dt": _set_dt, "grid": _new_grid}


@pytest.mark.parametrize("forced", [False, True])
@pytest.mark.parametrize("what", list(CHANGES))
@pytest.mark.parametrize("precision, persistent", [("fp32", 0), ("fp32", 256), ("fp64", 0)])
def test_member_changed_between_batch_calls(precision, persistent, what, forced):
    import __graft_entry__ as g
    g.build()
    from raytracer_3d_gb300.batch import Batch
    exps = [configs.shear_mini(n=n, seed=50 + i)
            for i, n in enumerate([(8, 8, 8, 4, 4, 4), (6, 5, 6, 4, 4, 6), (32, 16, 4, 4, 2, 4)])]

    def make(e):
        m = configs.build_model(e, precision)
        if forced:
            F = np.random.default_rng(7).random(m.forcing_shape()) * 1e-4
            m.set_forcing("flux", np.asfortranarray(F))
        return m

    alone = []
    for j, e in enumerate(exps):
        m = make(e)
        m.integrate(3)
        m.sync()
        if j != 1:
            CHANGES[what](m, e)
        m.integrate(5)
        alone.append(m.get_state().copy())
        m.close()
    models = [make(e) for e in exps]
    b = Batch(models)
    b.set_tuning(4, 256, 0, 4)
    b.set_persistent(persistent)
    b.integrate(3)
    b.sync()
    for j, (m, e) in enumerate(zip(models, exps)):
        if j != 1:
            CHANGES[what](m, e)
    b.integrate(5)          # a graph and a single launch
    for e, m, ref in zip(exps, models, alone):
        sl = interior(e.n)
        assert np.array_equal(m.get_state()[sl], ref[sl]), e.n
    b.close()
    for m in models:
        m.close()
