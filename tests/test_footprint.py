"""The device memory that the serving loop charges for a request is what its
member holds and what its set-up takes."""
import pytest

from harness import configs
from raytracer_3d_gb300.serve import GpuExecutor, Request, bytes_per_cell

SHAPES = [(4,) * 6, (8,) * 6, (8, 8, 8, 8, 8, 12), (16, 16, 8, 8, 8, 8), (6, 5, 7, 2, 4, 6), (1, 1, 40, 1, 1, 120),
          (33, 20, 8, 2, 10, 30), (24, 24, 24, 12, 12, 16)]


@pytest.fixture(scope="module", autouse=True)
def _built():
    import __graft_entry__ as g
    g.build_library()


def _footprint(n, precision):
    e = configs.shear_mini(n=n)
    return GpuExecutor(precision).footprint(Request(0, e, 1, 0.0, cells=e.cells))


def test_kept_and_transient_scratch_are_charged():
    # 10.2 MB of fields and 8.5 MB of scratch that stays with a small member
    res, tmp = _footprint((8,) * 6, "fp32")
    assert 18.6e6 < res < 20e6 and tmp == 0
    # a large one holds its fields and tables; its set-up takes a ring of at most 256 MB
    n = (24, 24, 24, 12, 12, 16)
    res, tmp = _footprint(n, "fp32")
    cells = 24 ** 3 * 12 * 12 * 16
    assert 36 * cells < res < 42 * cells
    assert 0 < tmp <= 256 << 20
    # the largest members: three m planes of the relation and of 1/omega
    n = (32, 32, 32, 24, 24, 24)
    plane = 33 ** 3 * 26 ** 2 + 32 ** 3 * 24 ** 2
    assert _footprint(n, "fp32")[1] == 3 * 8 * plane


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_per_cell_figures_bound_larger_members(precision):
    per = sum(bytes_per_cell(precision))
    for n in [(4,) * 6, (8,) * 6, (16,) * 6, (32, 32, 32, 24, 24, 24), (8, 32, 16, 8, 24, 12)]:
        cells = 1
        for k in n:
            cells *= k
        assert sum(_footprint(n, precision)) <= per * cells


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n", SHAPES)
def test_footprint_is_what_the_member_holds(n, precision):
    exp = configs.shear_mini(n=n)
    exp.fixed = (1e-3, 0.0, 1e-2)
    m = configs.build_model(exp, precision, padded=False)
    m.set_state()
    m.integrate(1)
    assert m.device_bytes() == _footprint(n, precision)[0]
    m.close()
