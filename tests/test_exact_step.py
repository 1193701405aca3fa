"""The bit-exact binary64 step without binary64 divisions: its integer
quotient against the division instruction (host, and on the GPU), and its
two forms against the one-thread-per-cell kernel, which the parity tests
hold to the oracle, at the edges of their ranges."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from harness import ROOT, configs

SRC = os.path.join(ROOT, "tests", "native", "exact_div_check.cu")


def _check(tmp_path, *args, flags=(), src=SRC):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "exact_div_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17", *flags,
                    "-I" + os.path.join(ROOT, "raytracer_3d_gb300", "csrc"), "-o", exe, src], check=True)
    r = subprocess.run([exe, *args], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("ulp", ["0", "1u", "0xffffffffu"])
def test_integer_quotient_on_the_host(tmp_path, ulp):
    _check(tmp_path, flags=("-DRT_RECIP_HOST_ULP=" + ulp,))


@pytest.mark.gpu
def test_integer_quotient_on_the_gpu(tmp_path):
    _check(tmp_path, "--device")


@pytest.mark.gpu
@pytest.mark.parametrize("walls", [True, False])
@pytest.mark.parametrize("n", [
    (4, 4, 4, 8, 8, 16), (4, 4, 4, 8, 8, 18),     # last field of one launch, first of two passes
    (16, 16, 16, 8, 8, 18), (15, 7, 12, 10, 12, 16),   # slabs over m; the last one shorter
    (16, 16, 64, 2, 140, 1),                      # over l, and several of them
    (160, 128, 110, 1, 1, 1), (2100, 1100, 1, 1, 1, 1),   # over z (its own face-0 plane) and y
])
def test_forms_equal_the_cell_kernel(n, walls):
    import __graft_entry__ as g
    g.build()
    rng = np.random.default_rng(5)
    exp = configs.shear_mini(n=n, upper=walls, lower=walls)
    exp.fixed = (1e-3, 0.0, 1e-2)     # wavenumbers of collapsed axes
    got = []
    E0 = rng.random(n) ** 4 * 1e-3
    for variant in ("cell", "tma", "split"):
        m = configs.build_model(exp, "fp64")
        m.E[(slice(2, -2),) * 6] = E0
        m.set_state()
        m.set_tuning(variant, 8, 256)
        m.integrate(3)
        got.append(m.get_state()[(slice(2, -2),) * 6].copy())
        m.close()
    assert np.isfinite(got[0]).all()
    assert np.array_equal(got[1], got[0]) and np.array_equal(got[2], got[0])


@pytest.mark.gpu
@pytest.mark.parametrize("walls", [True, False])
@pytest.mark.parametrize("forcing", ["none", "flux", "relax"])
@pytest.mark.parametrize("n", [(1, 1, 40, 1, 1, 120), (6, 5, 6, 4, 4, 6), (2, 2, 2, 2, 2, 2), (1, 9, 6, 1, 12, 100),
                               (7, 3, 5, 2, 6, 4), (1, 1, 2, 1, 1, 4), (300, 1, 1, 8, 1, 2)])
def test_many_steps_in_one_launch(n, forcing, walls):
    """nine steps in one launch, and as launches of one step, against the
    one-thread-per-cell kernel with its forcing kernel before every step"""
    import __graft_entry__ as g
    g.build()
    rng = np.random.default_rng(6)
    exp = configs.shear_mini(n=n, upper=walls, lower=walls)
    exp.fixed = (1e-3, 0.0, 1e-2)
    E0 = rng.random(n) ** 4 * 1e-3
    sl = (slice(2, -2),) * 6
    got = []
    for variant, parts in (("cell", (9,)), ("tma", (9,)), ("tma", (1,) * 9), ("tma", (4, 5))):
        m = configs.build_model(exp, "fp64")
        m.E[sl] = E0
        m.set_state()
        if forcing != "none":
            m.set_forcing(forcing, np.asfortranarray(np.random.default_rng(7).random(m.forcing_shape()) * 1e-4))
        m.set_tuning(variant, 8, 256)
        l0 = m.launch_count()
        for k in parts:
            m.integrate(k)
        launches = m.launch_count() - l0
        E = m.get_state()[sl].copy()
        b, f = m.diagnose()
        got.append((E, [b["eint"], b["mflint"], b["mfl_max"]] + [f[q].copy() for q in sorted(f)]))
        m.close()
        if variant == "tma":
            assert launches == (len(parts) if len(parts) < 9 else (9 if forcing == "none" else 18))
    for E, b in got[1:]:
        assert np.array_equal(E, got[0][0])
        assert all(np.array_equal(x, y) for x, y in zip(b, got[0][1]))


@pytest.mark.gpu
def test_integer_differences_on_the_gpu(tmp_path):
    _check(tmp_path, src=os.path.join(ROOT, "tests", "native", "flux_near_check.cu"))


FLOAT = os.path.join(ROOT, "tests", "native", "float_rn_check.cu")


def test_conversion_to_binary32_on_the_host(tmp_path):
    _check(tmp_path, src=FLOAT)


@pytest.mark.gpu
def test_conversion_to_binary32_on_the_gpu(tmp_path):
    _check(tmp_path, "--device", src=FLOAT)


SQRT = os.path.join(ROOT, "tests", "native", "sqrt_rn_check.cu")


@pytest.mark.parametrize("ulp", ["0", "2u", "0xfffffffeu"])
def test_square_root_on_the_host(tmp_path, ulp):
    _check(tmp_path, src=SQRT, flags=("-DRT_RECIP_HOST_ULP=" + ulp,))


@pytest.mark.gpu
def test_square_root_on_the_gpu(tmp_path):
    _check(tmp_path, "--device", src=SQRT)


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -262])   # the second: next to the end of the integer range
@pytest.mark.parametrize("n", [(16, 16, 64, 2, 70, 1), (15, 7, 12, 10, 12, 16)])
def test_near_and_far_values_equal_the_cell_kernel(n, scale):
    """most warps take the integer differences, those around the rough and the zero cells do not"""
    import __graft_entry__ as g
    g.build()
    rng = np.random.default_rng(6)
    exp = configs.shear_mini(n=n)
    exp.fixed = (1e-3, 0.0, 1e-2)
    sl = (slice(2, -2),) * 6
    E0 = scale * (1 + 3 * rng.random(n))
    E0[:, :, n[2] // 2, 0] *= rng.random(n)[:, :, n[2] // 2, 0] ** 20
    E0[0, 0, 0] = 0.0
    got = []
    for variant in ("cell", "split"):
        m = configs.build_model(exp, "fp64")
        m.E[sl] = E0
        m.set_state()
        m.set_tuning(variant, 8, 256)
        m.integrate(3)
        got.append(m.get_state()[sl].copy())
        m.close()
    assert np.array_equal(got[0].view(np.uint64), got[1].view(np.uint64))
