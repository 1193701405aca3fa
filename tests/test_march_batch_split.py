"""The members of a binary32 batch over launches, on the host (no GPU needed)."""
import os
import shutil
import subprocess

import pytest

from harness import ROOT


def test_members_per_launch(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    import __graft_entry__ as g
    g.build_library()
    pkg = os.path.join(ROOT, "raytracer_3d_gb300")
    exe = str(tmp_path / "march_batch_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17", "-cudart", "shared",
                    "-I" + os.path.join(pkg, "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "native", "march_batch_check.cu"),
                    "-L" + pkg, "-lraytracer_gb300", "-Xlinker", "-rpath=" + pkg], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
