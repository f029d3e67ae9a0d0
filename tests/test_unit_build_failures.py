"""The unit layout's build when one of its calls fails, on the CPU over a faked CUDA runtime: see
tests/cpp/unit_build_failures.cu."""
import os
import shutil
import subprocess

import pytest

CPP = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp")


def test_nothing_is_queued_behind_a_failure(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path / "unit_build_failures")
    cmd = [nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "--expt-relaxed-constexpr",
           "-Xptxas", "-O0", "--cudart=none", os.path.join(CPP, "unit_build_failures.cu"),
           os.path.join(CPP, "fake_cudart.cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
    allocations, calls = (int(x) for x in r.stdout.split()[1:])
    assert allocations > 30 and calls > 20  # the build went to its end
