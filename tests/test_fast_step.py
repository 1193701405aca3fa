"""The fast binary64 step: its integer slopes against the direct ones (host
and GPU), and the step over several slabs against the bit-exact one."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from harness import ROOT, configs, max_rel

SRC = os.path.join(ROOT, "tests", "native", "slope_near_check.cu")


def _check(tmp_path, *args):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "slope_near_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17",
                    "-I" + os.path.join(ROOT, "raytracer_3d_gb300", "csrc"), "-o", exe, SRC], check=True)
    r = subprocess.run([exe, *args], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def test_integer_slopes_on_the_host(tmp_path):
    _check(tmp_path)


@pytest.mark.gpu
def test_integer_slopes_on_the_gpu(tmp_path):
    _check(tmp_path, "--device")


@pytest.mark.gpu
@pytest.mark.parametrize("walls", [True, False])
@pytest.mark.parametrize("n, stretched", [
    ((16, 16, 16, 8, 8, 18), False),      # three slabs, rows within a warp, one spacing per axis
    ((15, 7, 12, 10, 12, 16), True),      # two slabs, ragged rows, varying spacings
    ((160, 128, 110, 2, 1, 1), False),    # a slab of one volume
    ((33, 20, 8, 2, 30, 30), False),      # rings of k and l longer than a slab's share
])
def test_slabs_against_the_exact_step(n, stretched, walls):
    import __graft_entry__ as g
    g.build()
    make = configs.stretched_mini if stretched else configs.shear_mini
    exp = make(n=n, upper=walls, lower=walls)
    exp.fixed = (1e-3, 0.0, 1e-2)
    rng = np.random.default_rng(8)
    sl = (slice(2, -2),) * 6
    # smooth in most of the field, rough (far from the integer range, and zero) in a corner
    E0 = 1e-3 * (1 + rng.random(n))
    E0[: n[0] // 2, :, :, 0] *= rng.random(n)[: n[0] // 2, :, :, 0] ** 20
    E0[0, 0] = 0.0
    got = []
    for variant in ("split", "fast"):
        m = configs.build_model(exp, "fp64")
        m.E[sl] = E0
        m.set_state()
        m.set_tuning(variant, 8, 256)
        out = []
        for _ in range(3):
            m.integrate(1)
            out.append(m.get_state()[sl].copy())
        got.append(out)
        m.close()
    for step, (a, b) in enumerate(zip(*got)):
        assert max_rel(b, a) <= 1e-12 * (step + 1), step
