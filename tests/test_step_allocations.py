"""Steps allocate nothing: what a handle works with is there once its
coefficients and schedule are, so the first step can be captured."""
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
