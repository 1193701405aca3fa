"""Set-up calls and rebuilds of a batch right behind queued steps: the steps
still see the tables they were queued with, and the next ones the new ones."""
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


@pytest.mark.parametrize("precision, persistent", [("fp32", 0), ("fp32", 256), ("fp64", 0)])
def test_rebuild_does_not_reach_queued_batch_steps(precision, persistent):
    """a member stepped on its own flips its buffers, so the batch builds its
    member arrays anew while its earlier launches may still read them"""
    import __graft_entry__ as g
    g.build()
    from raytracer_3d_gb300.batch import Batch
    exps = [configs.shear_mini(n=n, seed=60 + i) for i, n in enumerate([(32, 32, 16, 4, 4, 8), (8, 8, 16, 4, 4, 8)])]
    got = []
    for wait in (True, False):
        models = [configs.build_model(e, precision, padded=False) for e in exps]
        for m in models:
            m.set_state()
        b = Batch(models)
        b.set_tuning(4, 256, 0, 4)
        b.set_persistent(persistent)
        for _ in range(4):
            b.integrate(41)
            if wait:
                b.sync()
            models[1].integrate(1)
            if wait:
                models[1].sync()
        b.integrate(3)
        got.append([m.get_state() for m in models])
        b.close()
        for m in models:
            m.close()
    for x, y in zip(*got):
        assert np.isfinite(x).all() and np.array_equal(x, y)
