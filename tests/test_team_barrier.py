"""The team barrier's withdrawal, checked on the host against every moment at
which the rest of the team may go on (tests/cxx/team_barrier.cu, compiled by
nvcc as host code)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_withdrawal_leaves_the_next_generation_alone(tmp_path):
    nvcc = next((c for c in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc")
                 if c and os.path.exists(c)), None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "team_barrier")
    build = subprocess.run([nvcc, "-std=c++17", "-O2", "-x", "cu", "-I" + os.path.join(ROOT, "213transpose_b200", "csrc"),
                            os.path.join(ROOT, "tests", "cxx", "team_barrier.cu"), "-o", exe], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0 and run.stdout.startswith("ok"), run.stdout + run.stderr
