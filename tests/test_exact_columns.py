"""Columns of tens of thousands of cells, many steps in one launch: the forms
of exact_small_kernel that keep two faces, one face or nothing per thread in
registers, on both sides of each limit, against the one-thread-per-cell kernel."""
import numpy as np
import pytest

from harness import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walls", [True, False])
@pytest.mark.parametrize("forcing", ["none", "flux", "relax"])
@pytest.mark.parametrize("n", [
    (1, 1, 160, 1, 1, 300),     # open walls: 793 faces per CTA on 152 SMs, two per thread; reflecting: 1109, none kept
    (1, 1, 64, 1, 1, 1024),     # the largest field of one launch
    (1, 1, 80, 1, 1, 260),      # about 500 faces: one per thread or two
    (1, 1, 3, 1, 1, 20000), (40, 1, 1, 1000, 1, 1),
])
def test_columns_equal_the_cell_kernel(n, forcing, walls):
    if forcing != "none" and n[2] == 1:
        pytest.skip("a forcing acts on the bottom of a z axis")
    import __graft_entry__ as g
    g.build()
    exp = configs.shear_mini(n=n, upper=walls, lower=walls)
    exp.fixed = (1e-3, 0.0, 1e-2)
    E0 = np.random.default_rng(6).random(n) ** 4 * 1e-3
    sl = (slice(2, -2),) * 6
    got = []
    for variant, parts in (("cell", (11,)), ("tma", (11,)), ("tma", (5, 6))):
        m = configs.build_model(exp, "fp64")
        m.E[sl] = E0
        m.set_state()
        if forcing != "none":
            m.set_forcing(forcing, np.asfortranarray(np.random.default_rng(7).random(m.forcing_shape()) * 1e-4))
        m.set_tuning(variant, 8, 256)
        l0 = m.launch_count()
        for k in parts:
            m.integrate(k)
        if variant == "tma":
            assert m.launch_count() - l0 == len(parts)
        got.append(m.get_state()[sl].copy())
        m.close()
    assert np.isfinite(got[0]).all() and got[0].any()
    for E in got[1:]:
        assert np.array_equal(E, got[0])
