"""A ragged plan whose bands cannot be launched, on the host
(tests/cxx/ragged_refusal.cu, compiled by nvcc with the launcher's neighbours
stubbed): no other plan may run on a tensor whose segments have moved."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_refusal_after_the_walk_is_an_error(tmp_path):
    nvcc = next((c for c in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc")
                 if c and os.path.exists(c)), None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "ragged_refusal")
    build = subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                            "-I" + os.path.join(ROOT, "213transpose_b200", "csrc"), "-I" + os.path.join(ROOT, "include"),
                            os.path.join(ROOT, "tests", "cxx", "ragged_refusal.cu"), "-o", exe], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0 and run.stdout.startswith("ok"), run.stdout + run.stderr
