"""The binary32 march at exactly 2^30 cells, the largest field it takes (32-bit
byte offsets into E): the bench's 32^6 workload, two steps, against the staged
z march and, its limit taken away, the TMA plane kernel, bit for bit."""
import dataclasses

import numpy as np
import pytest

from harness import configs

pytestmark = pytest.mark.gpu


def test_march_at_two_to_the_30_cells():
    import __graft_entry__ as g
    g.build()
    exp = configs.jet_large()
    assert exp.cells == 1 << 30
    m = configs.build_model(exp, "fp32", padded=False)
    try:
        E0 = np.asfortranarray(m.E, dtype=np.float32)
        m.E = E0
        m.set_state()
        m.integrate(2)
        want = m.get_state()
        assert np.isfinite(want).all() and not np.array_equal(want, E0)
    finally:
        m.close()
    # new handles: the steps of each draw the same random words
    exp = dataclasses.replace(exp, initial=lambda m, rng: None)
    for variant, fallback in (("w2z", 0), ("tma", 1)):
        m = configs.build_model(exp, "fp32", padded=False)
        try:
            m.E = E0
            m.set_state()
            m.set_tuning(variant, 8, 512, 1)
            m._check(m._lib.rt_selftest_fallback(m.handle, fallback), "rt_selftest_fallback")
            m.integrate(2)
            got = m.get_state()
        finally:
            m.close()
        assert np.array_equal(got, want), variant
