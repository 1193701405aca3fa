"""The kernels whose shared memory depends on the field: a handle or a batch of
small planes leaves the launches of large ones as they were."""
import threading

import numpy as np
import pytest

from harness import configs

pytestmark = pytest.mark.gpu

LARGE, SMALL = (24, 24, 6, 2, 2, 4), (8, 8, 6, 2, 2, 4)


def _model(n, precision):
    m = configs.build_model(configs.shear_mini(n=n), precision, padded=False)
    m.set_state()
    return m


def _alone(n, precision, steps):
    m = _model(n, precision)
    m.set_tuning("cell", 8, 256)
    m.integrate(steps)
    E = m.get_state()
    m.close()
    return E


@pytest.mark.parametrize("precision, persistent", [("fp64", 0), ("fp32", 256)])
def test_batches_of_large_and_small_planes(precision, persistent):
    import __graft_entry__ as g
    g.build()
    from raytracer_3d_gb300.batch import Batch
    models = [_model(n, precision) for n in (LARGE, SMALL)]
    batches = [Batch([m]) for m in models]
    for b in batches:
        b.set_tuning(4, 256, 0, 2)
        b.set_persistent(persistent)
    for _ in range(3):
        for b in batches:
            b.integrate(1)
    for b in batches:
        b.sync()
    for n, m in zip((LARGE, SMALL), models):
        assert np.array_equal(m.get_state(), _alone(n, precision, 3)), n
    for b in batches:
        b.close()
    for m in models:
        m.close()


@pytest.mark.parametrize("precision, variant", [("fp64", "group"), ("fp32", "group"), ("fp32", "w3"), ("fp32", "w6")])
def test_two_host_threads(precision, variant):
    import __graft_entry__ as g
    g.build()
    steps = 1500
    models = [_model(n, precision) for n in (LARGE, SMALL)]
    errors = []

    def run(m):
        try:
            for _ in range(steps):
                m.integrate(1)
        except Exception as e:
            errors.append(e)

    for m in models:
        m.set_tuning(variant, 8, 256)
    threads = [threading.Thread(target=run, args=(m,)) for m in models]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    for n, m in zip((LARGE, SMALL), models):
        assert np.array_equal(m.get_state(), _alone(n, precision, steps)), n
        m.close()
