"""Coefficients of a field whose dispersion relation does not fit the scratch
at once (it is evaluated in batches of m planes): a step's cells against the
per-cell oracle, the CFL rate against the velocities, bit for bit."""
import numpy as np
import pytest

from harness import ONX, build_point_oracle, configs, sample_cells

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walls", [True, False])
def test_batches_of_m_planes(walls):
    import __graft_entry__ as g
    g.build()
    n = (40, 40, 2, 20, 20, 8)          # 30 MB a plane: batches of seven planes and one
    exp = configs.shear_mini(n=n, upper=walls, lower=walls)
    m = configs.build_model(exp, "fp64")
    po = None
    try:
        sl = (slice(ONX, -ONX),) * 6
        E0 = np.asfortranarray(np.random.default_rng(3).random(n) * 1e-3)
        m.E[sl] = E0
        m.set_state()
        m.integrate(1)
        E1 = m.get_state()[sl]
        po = build_point_oracle(exp, m.dt)
        cells = sample_cells(n, 3000, np.random.default_rng(4))
        assert np.array_equal(E1[tuple((cells - 1).T)], po.point_steps(E0, cells))
        rate = np.zeros(n)
        for a, ax in enumerate("xyzklm"):
            v = np.abs(m.get_field(a))
            lo, hi = list(sl), list(sl)
            lo[a] = slice(ONX - 1, -ONX - 1)
            d = m.grid[ax]["dt"][ONX:-ONX].reshape([-1 if b == a else 1 for b in range(6)])
            rate = rate + np.maximum(v[tuple(lo)], v[tuple(hi)]) / d
        assert m.max_rate() == rate.max()
    finally:
        if po is not None:
            po.close()
        m.close()
