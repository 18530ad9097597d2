"""Every width of the kernels' generator window, and its draws without checks,
against the lazily computed Philox stream on the host (rng_draws_check.cu, which
includes the engine's own header)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_unchecked_draws_match_the_lazy_stream(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = tmp_path / "rng_draws_check"
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "egsnrc_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "rng_draws_check.cu"), "-o", str(exe)],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("ok")
    assert all(int(x) > 100000 for x in r.stdout.split()[1:4])
