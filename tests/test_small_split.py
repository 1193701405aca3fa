"""The one-launch binary64 step: its shared memory stays below what a launch may
have without raising the kernel's limit, on any GPU, and so two host threads
that step fields of different sizes do not get in each other's way."""
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest

from harness import ROOT, configs


def test_split_fits_without_an_attribute(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    import __graft_entry__ as g
    g.build_library()
    pkg = os.path.join(ROOT, "raytracer_3d_gb300")
    exe = str(tmp_path / "small_split_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17", "-I" + os.path.join(pkg, "csrc"),
                    "-o", exe, os.path.join(ROOT, "tests", "native", "small_split_check.cu"), "-L" + pkg,
                    "-lraytracer_gb300", "-Xlinker", "-rpath=" + pkg], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
def test_two_host_threads_step_fields_of_different_sizes():
    import __graft_entry__ as g
    g.build()
    shapes = [(2, 2, 2, 2, 2, 2), (8, 8, 8, 4, 4, 8)]
    steps = 4000

    def start(n):
        m = configs.build_model(configs.shear_mini(n=n), "fp64", padded=False)
        m.set_state()
        return m

    alone = []
    for n in shapes:
        m = start(n)
        for _ in range(steps):
            m.integrate(1)
        alone.append(m.get_state())
        m.close()
    models = [start(n) for n in shapes]
    errors = []

    def run(m):
        try:
            for _ in range(steps):
                m.integrate(1)
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=run, args=(m,)) for m in models]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    for m, want in zip(models, alone):
        assert np.array_equal(m.get_state(), want)
        m.close()
