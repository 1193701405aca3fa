"""The binary32 step of threads marching along k against the one-thread-per-
cell kernel, bit for bit: vector widths 4, 2 and 1, rows and planes that end
inside a CTA, walks in segments, short last bands, collapsed axes, both
walls; and a batch of more members than one launch takes."""
import numpy as np
import pytest

from harness import configs

pytestmark = pytest.mark.gpu


def _state(n, seed):
    r = np.random.default_rng(seed)
    return np.asfortranarray((r.random(n) ** 6 * 1e-3).astype(np.float32))


def _model(n, walls, E):
    exp = configs.shear_mini(n=n, upper=walls, lower=walls)
    exp.fixed = (1e-3, 0.0, 1e-2)
    m = configs.build_model(exp, "fp32", padded=False)
    m.E = E
    m.set_state()
    return m


@pytest.mark.parametrize("walls", [True, False])
@pytest.mark.parametrize("n", [
    (4, 2, 2, 2, 2, 2), (6, 3, 5, 4, 2, 6), (7, 3, 5, 2, 6, 4), (2, 2, 2, 2, 2, 2), (1, 6, 8, 4, 6, 4),
    (8, 8, 4, 6, 2, 10), (12, 11, 2, 8, 4, 2), (32, 32, 3, 2, 2, 2), (5, 1, 8, 4, 1, 6), (16, 5, 1, 6, 2, 1),
    (9, 4, 6, 1, 4, 4), (1, 1, 10, 1, 1, 12), (260, 2, 2, 2, 2, 2),
])
def test_march_equals_the_cell_kernel(n, walls):
    import __graft_entry__ as g
    g.build()
    E = _state(n, 1)
    ref = _model(n, walls, E)
    ref.set_tuning("cell", 8, 256)
    ref.integrate(3)
    want = ref.get_state()
    ref.close()
    for variant, band, sweep in (("tma", 8, 0), ("tma", 3, 1), ("w2q", 1, 0)):
        m = _model(n, walls, E)
        m.set_tuning(variant, band, 512, sweep)
        m.integrate(3)
        assert np.array_equal(m.get_state(), want), (variant, band, sweep)
        m.close()


def test_batch_of_many_members():
    import __graft_entry__ as g
    g.build()
    from raytracer_3d_gb300.batch import Batch
    shapes = [(4, 4, 4, 2, 2, 2), (6, 3, 4, 2, 4, 2), (5, 4, 2, 4, 2, 2), (8, 8, 8, 4, 2, 4)]
    want = {n: None for n in shapes}
    for n in shapes:
        m = _model(n, True, _state(n, 2))
        m.set_tuning("cell", 8, 256)
        m.integrate(5)
        want[n] = m.get_state()
        m.close()
    models = [_model(shapes[j % 4], True, _state(shapes[j % 4], 2)) for j in range(83)]
    b = Batch(models)
    b.set_tuning(4, 256, 0, 2)
    b.integrate(2)
    b.integrate(3)
    assert b.launch_count() == 10          # 80 members and 3
    for j, m in enumerate(models):
        assert np.array_equal(m.get_state(), want[shapes[j % 4]]), j
    b.close()
    for m in models:
        m.close()
