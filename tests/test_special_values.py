"""States with infinities, NaN, denormals, huge, negative and signed-zero
values: the steps that keep the reference's arithmetic give what the
one-thread-per-cell kernel gives, value for value (NaN for NaN)."""
import numpy as np
import pytest

from harness import configs

pytestmark = pytest.mark.gpu


def _state(n, dtype, kinds, seed):
    r = np.random.default_rng(seed)
    E = (r.random(n) ** 6 * 1e-3).astype(dtype)
    tiny = float(np.finfo(dtype).smallest_subnormal)
    huge = float(np.finfo(dtype).max)
    values = {"denormal": [tiny, 7 * tiny, -3 * tiny, float(np.finfo(dtype).tiny)], "zero": [0.0, -0.0],
              "huge": [huge, -huge, 0.6 * huge, 1e-3 * huge], "inf": [np.inf, -np.inf], "nan": [np.nan],
              "negative": [-1e-3, -1e-9]}
    pool = np.array([v for k in kinds for v in values[k]], dtype=dtype)
    at = r.random(n) < 0.05
    E[at] = r.choice(pool, size=int(at.sum()))
    return np.asfortranarray(E)


def _run(n, precision, walls, E, variant, steps, fallback=0):
    exp = configs.shear_mini(n=n, upper=walls, lower=walls)
    exp.fixed = (1e-3, 0.0, 1e-2)
    m = configs.build_model(exp, precision, padded=False)
    m.E = E
    m.set_state()
    m.set_tuning(variant, 8, 256)
    m._check(m._lib.rt_selftest_fallback(m.handle, fallback), "rt_selftest_fallback")
    for k in steps:
        m.integrate(k)
    out = m.get_state()
    m.close()
    return out


@pytest.mark.parametrize("kinds", [("denormal", "zero"), ("negative", "zero", "huge"), ("inf",), ("nan",),
                                   ("denormal", "zero", "huge", "inf", "nan", "negative")])
@pytest.mark.parametrize("precision, n", [
    ("fp64", (6, 5, 6, 4, 4, 6)), ("fp64", (1, 1, 40, 1, 1, 120)), ("fp64", (16, 8, 8, 6, 4, 6)),
    ("fp64", (15, 7, 12, 4, 4, 6)), ("fp32", (8, 5, 6, 4, 4, 6)), ("fp32", (6, 5, 6, 4, 4, 6)), ("fp32", (7, 3, 5, 2, 6, 4))])
def test_special_values_equal_the_cell_kernel(precision, n, kinds):
    import __graft_entry__ as g
    g.build()
    E = _state(n, np.float64 if precision == "fp64" else np.float32, kinds, 9)
    for walls in (True, False):
        want = _run(n, precision, walls, E, "cell", (4,))
        assert ("nan" in kinds) == bool(np.isnan(_run(n, precision, walls, E, "cell", ())).any())
        for steps in ((4,), (1, 1, 1, 1)):
            got = _run(n, precision, walls, E, "tma", steps)
            assert np.array_equal(got, want, equal_nan=True), (walls, steps)


@pytest.mark.parametrize("kinds", [("denormal", "zero"), ("negative", "zero", "huge"), ("inf",), ("nan",)])
@pytest.mark.parametrize("n", [(16, 8, 8, 6, 4, 6), (15, 7, 12, 4, 4, 6)])
def test_special_values_in_the_plane_kernels(n, kinds):
    import __graft_entry__ as g
    g.build()
    from raytracer_3d_gb300.batch import Batch
    E = _state(n, np.float64, kinds, 9)
    want = _run(n, "fp64", False, E, "cell", (3,))
    for variant, fallback in (("plane", 0), ("group", 0), ("tma", 1)):
        assert np.array_equal(_run(n, "fp64", False, E, variant, (3,), fallback), want, equal_nan=True), variant
    exp = configs.shear_mini(n=n, upper=False, lower=False)
    exp.fixed = (1e-3, 0.0, 1e-2)
    m = configs.build_model(exp, "fp64", padded=False)
    m.E = E
    m.set_state()
    b = Batch([m])
    b.integrate(3)
    b.sync()
    assert np.array_equal(m.get_state(), want, equal_nan=True)
    b.close()
    m.close()


@pytest.mark.parametrize("kinds", [("denormal", "zero"), ("negative", "zero", "huge")])
@pytest.mark.parametrize("n", [(6, 5, 6, 4, 4, 6), (3, 4, 5, 10, 2, 6), (1, 1, 12, 1, 1, 20)])
def test_edge_integrals_of_special_values(n, kinds):
    """the budget's wavenumber integrals, edge fluxes among them, against the kernels that need no scratch"""
    import __graft_entry__ as g
    g.build()
    got = []
    for fallback in (0, 1):
        exp = configs.shear_mini(n=n, upper=False, lower=False)
        exp.fixed = (1e-3, 0.0, 1e-2)
        m = configs.build_model(exp, "fp64", padded=False)
        m._check(m._lib.rt_selftest_fallback(m.handle, fallback), "rt_selftest_fallback")
        m.E = _state(n, np.float64, kinds, 10)
        m.set_state()
        m.integrate(1)
        got.append(m.diagnose()[1])
        m.close()
    for k in got[0]:
        assert np.array_equal(got[0][k], got[1][k], equal_nan=True), k
