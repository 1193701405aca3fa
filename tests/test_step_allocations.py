"""Steps allocate nothing: what a handle works with is there once its
coefficients and schedule are, so the first step can be captured.  Scratch
that a handle can do without makes room for what a call cannot."""
import numpy as np
import pytest

from harness import configs

pytestmark = pytest.mark.gpu

SMALL, SLABS = (6, 5, 6, 4, 4, 6), (16, 16, 16, 6, 6, 8)


def _model(n, precision):
    m = configs.build_model(configs.shear_mini(n=n), precision, padded=False)
    m.set_state()
    return m


@pytest.mark.parametrize("schedules", [(), ("split",), ("fast",), ("plane",), ("cell", "tma"), ("fast", "split")])
@pytest.mark.parametrize("precision, n", [("fp64", SMALL), ("fp64", SLABS), ("fp32", SLABS)])
def test_first_step_allocates_nothing(precision, n, schedules):
    import __graft_entry__ as g
    g.build()
    m = _model(n, precision)
    for s in schedules:
        m.set_tuning(s, 8, 256)
    held = m.device_bytes()
    m.integrate(1)
    m.integrate(5)
    m.sync()
    assert m.device_bytes() == held
    m.close()


@pytest.mark.parametrize("precision, schedule, n, steps", [
    ("fp64", "tma", SMALL, 2), ("fp64", "tma", SMALL, 6), ("fp64", "split", SLABS, 2), ("fp64", "cell", SLABS, 2),
    ("fp32", "tma", SLABS, 2)])
def test_first_step_under_capture(precision, schedule, n, steps):
    import __graft_entry__ as g
    g.build()
    torch = pytest.importorskip("torch")
    ref = _model(n, precision)
    ref.set_tuning("cell", 8, 256)
    ref.integrate(2 * steps)
    want = ref.get_state()
    ref.close()
    m = _model(n, precision)
    m.set_tuning(schedule, 8, 256)
    m.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(torch.cuda.ExternalStream(m.stream())):
        graph.capture_begin(capture_error_mode="global")
        try:
            m.integrate(steps)      # an even number: the buffers end where they began
        finally:
            graph.capture_end()
        graph.replay()
        graph.replay()
    m.sync()
    assert np.array_equal(m.get_state(), want)
    m.close()


def test_scratch_makes_room():
    """rt_get_tendency beside a full GPU: its two fields fit only where the
    scratch of the steps and budgets was; later steps have theirs again"""
    import __graft_entry__ as g
    g.build()
    torch = pytest.importorskip("torch")
    n = (32, 32, 32, 8, 8, 16)
    m = configs.build_model(configs.shear_mini(n=n), "fp64")
    m.integrate(2)
    m.diagnose(fields=False)
    want = m.get_tendency()
    m.sync()
    held = m.device_bytes()
    need = 2 * 8 * 32 ** 3 * 1024
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    filler = torch.empty(free - need + (40 << 20), dtype=torch.uint8, device="cuda")
    got = m.get_tendency()
    assert all(np.array_equal(x, y) for x, y in zip(got, want))
    del filler
    torch.cuda.empty_cache()
    assert m.device_bytes() >= held - 16 * 2 ** 22      # all but the budget's
    m.integrate(1)
    b, _ = m.diagnose(fields=False)
    assert m.device_bytes() == held and np.isfinite(b["residual"])
    m.close()


def test_scratch_of_a_captured_step_stays():
    """a captured step holds the scratch's address: no call may give that
    scratch away while the graph can still be launched"""
    import __graft_entry__ as g
    g.build()
    torch = pytest.importorskip("torch")
    from raytracer_3d_gb300._lib import RtError
    n = (32, 32, 32, 8, 8, 16)
    ref = _model(n, "fp64")
    ref.integrate(6)
    want = ref.get_state()
    ref.close()
    m = _model(n, "fp64")
    m.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(torch.cuda.ExternalStream(m.stream())):
        graph.capture_begin(capture_error_mode="global")
        try:
            m.integrate(2)
        finally:
            graph.capture_end()
        graph.replay()
    m.integrate(2)
    m.sync()
    held = m.device_bytes()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    need = 2 * 8 * 32 ** 3 * 1024
    filler = torch.empty(free - need + (40 << 20), dtype=torch.uint8, device="cuda")
    with pytest.raises(RtError):
        m.get_tendency()
    assert m.device_bytes() == held
    del filler
    torch.cuda.empty_cache()
    with torch.cuda.stream(torch.cuda.ExternalStream(m.stream())):
        graph.replay()
    m.sync()
    assert np.array_equal(m.get_state(), want)
    m.close()


def test_fast_that_does_not_fit_leaves_all_as_it_was():
    """the fast step's fields on a full GPU: selection fails, and the handle
    holds what it held, the step's scratch included"""
    import __graft_entry__ as g
    g.build()
    torch = pytest.importorskip("torch")
    from raytracer_3d_gb300._lib import RtError
    n = (32, 32, 32, 8, 8, 16)
    ref = _model(n, "fp64")
    ref.integrate(3)
    want = ref.get_state()
    ref.close()
    m = _model(n, "fp64")
    m.integrate(1)
    m.sync()
    held = m.device_bytes()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    filler = torch.empty(free - (700 << 20), dtype=torch.uint8, device="cuda")    # two of its eight fields fit
    with pytest.raises(RtError):
        m.set_tuning("fast", 8, 256)
    assert m.device_bytes() == held
    m.integrate(2)
    assert np.array_equal(m.get_state(), want)
    del filler
    torch.cuda.empty_cache()
    m.set_tuning("fast", 8, 256)
    assert m.device_bytes() > held
    m.close()
