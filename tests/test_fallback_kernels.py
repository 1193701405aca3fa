"""The kernels that stand in where the usual ones cannot run (no memory for the
exact step's slabs and the budget's terms, or for the dispersion relation of
the coefficients; binary32 fields beyond the march), on small fields: the same
bits as the one-thread-per-cell kernel, and as the usual coefficients."""
import numpy as np
import pytest

from harness import configs

pytestmark = pytest.mark.gpu


def _model(n, precision, walls, fallback, seed=3):
    exp = configs.shear_mini(n=n, upper=walls, lower=walls)
    exp.fixed = (1e-3, 0.0, 1e-2)     # wavenumbers of collapsed axes
    m = configs.build_model(exp, precision, padded=False)
    m.E = np.asfortranarray(np.random.default_rng(seed).random(n) ** 4 * 1e-3)
    m.set_state()
    m._check(m._lib.rt_selftest_fallback(m.handle, int(fallback)), "rt_selftest_fallback")
    return m


def _cell(n, precision, walls, steps):
    m = _model(n, precision, walls, False)
    m.set_tuning("cell", 8, 256)
    m.integrate(steps)
    E = m.get_state()
    m.close()
    return E


@pytest.mark.parametrize("walls", [True, False])
@pytest.mark.parametrize("n, threads", [
    ((16, 16, 6, 8, 4, 6), 256), ((16, 16, 6, 8, 4, 6), 512),      # planes staged by TMA
    ((32, 32, 4, 4, 4, 4), 256),                                   # several cells per thread
    ((15, 7, 12, 4, 4, 6), 128),                                   # planes of plain loads: no multiple of 16 bytes
    ((2100, 1100, 1, 1, 1, 1), 256),                               # planes beyond shared memory
])
def test_binary64_without_scratch(n, threads, walls):
    import __graft_entry__ as g
    g.build()
    want = _cell(n, "fp64", walls, 3)
    usual = _model(n, "fp64", walls, False)
    usual.integrate(3)
    m = _model(n, "fp64", walls, True)
    held = m.device_bytes()
    assert held < usual.device_bytes()
    for variant in ("tma", "split"):
        m.set_state()
        m.set_tuning(variant, 8, threads)
        m.integrate(3)
        assert np.array_equal(m.get_state(), want), variant
    b, f = m.diagnose()
    assert m.device_bytes() == held
    bu, fu = usual.diagnose()
    for k in f:
        assert np.array_equal(f[k], fu[k]), k
    for k in b:
        if k in ("mfl_max", "umax", "vmax", "wmax", "kmax", "lmax", "mmax") or k.startswith("cfl"):
            assert b[k] == bu[k], k
    # sums of some 10^5 to 10^6 terms in two orders, against the largest of them
    scale = max(abs(bu[k]) for k in bu if k[:3] in ("ein", "mfl", "bfl"))
    for k in b:
        if k in ("eint", "mflint", "residual") or k.startswith("bfl"):
            assert abs(b[k] - bu[k]) <= 1e-12 * scale, k
    usual.close()
    m.close()


@pytest.mark.parametrize("walls", [True, False])
@pytest.mark.parametrize("variant, threads", [("tma", 256), ("tma", 512), ("w2q", 256), ("w2q", 512)])
@pytest.mark.parametrize("n", [(32, 32, 4, 4, 2, 4), (24, 16, 6, 4, 2, 4), (7, 3, 5, 2, 6, 4), (200, 130, 2, 2, 2, 2)])
def test_binary32_beyond_the_march(n, variant, threads, walls):
    import __graft_entry__ as g
    g.build()
    want = _cell(n, "fp32", walls, 3)
    m = _model(n, "fp32", walls, True)
    m.set_tuning(variant, 4, threads, 1)
    m.integrate(3)
    assert np.array_equal(m.get_state(), want)
    m.close()


@pytest.mark.parametrize("shapes", [
    [(32, 32, 4, 4, 2, 4), (16, 8, 4, 2, 2, 4)],     # z groups
    [(64, 40, 4, 2, 2, 2), (32, 32, 2, 2, 2, 2)],    # planes staged by TMA
    [(7, 3, 5, 2, 6, 4), (5, 4, 3, 2, 2, 2)],        # planes of plain loads
])
def test_batch_beyond_the_march(shapes):
    import __graft_entry__ as g
    g.build()
    from raytracer_3d_gb300.batch import Batch
    models = [_model(n, "fp32", True, True) for n in shapes]
    b = Batch(models)
    b.set_tuning(4, 256, 0, 2)
    b.integrate(2)
    b.integrate(3)
    for n, m in zip(shapes, models):
        assert np.array_equal(m.get_state(), _cell(n, "fp32", True, 5)), n
    for m in models:                                 # and back to the march, one launch for all
        m._check(m._lib.rt_selftest_fallback(m.handle, 0), "rt_selftest_fallback")
    l0 = b.launch_count()
    b.integrate(3)
    assert b.launch_count() - l0 == 3
    for n, m in zip(shapes, models):
        assert np.array_equal(m.get_state(), _cell(n, "fp32", True, 8)), n
    b.close()
    for m in models:
        m.close()


@pytest.mark.parametrize("walls", [True, False])
@pytest.mark.parametrize("n", [
    (6, 5, 6, 4, 4, 6), (16, 3, 7, 8, 2, 10), (5, 4, 3, 2, 1, 2), (1, 6, 8, 4, 6, 4), (9, 1, 6, 6, 4, 2),
    (1, 1, 12, 1, 1, 20), (40, 30, 1, 1, 1, 1),
])
def test_coefficients_without_scratch(n, walls):
    import __graft_entry__ as g
    g.build()
    m = _model(n, "fp64", walls, False)
    fields = [m.get_field(w) for w in range(9)]
    rate = m.max_rate()
    m.integrate(3)
    E = m.get_state()
    m.set_state()
    m._check(m._lib.rt_selftest_fallback(m.handle, 1), "rt_selftest_fallback")
    m.U *= 2.0                       # other coefficients first, so that nothing is left from before
    m.calc_parameter()
    m.U *= 0.5
    m.calc_parameter()
    assert m.max_rate() == rate
    for w, want in enumerate(fields):
        assert np.array_equal(m.get_field(w), want), w
    m.integrate(3)
    assert np.array_equal(m.get_state(), E)
    m.close()
