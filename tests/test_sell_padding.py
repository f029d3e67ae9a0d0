"""The sliced layout's slots of empty stencils name a row that their slice reads anyway, so that no
kernel reads a row of the source that the table does not name (sell.h).  The rule, which the device
build and this test compile from the same header, over tables with empty stencils anywhere and no
entry below row 100."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("no compiler or no CUDA headers")
    d = tmp_path_factory.mktemp("sell")
    src, lib = str(d / "rule.cpp"), str(d / "rule.so")
    with open(src, "w") as f:
        f.write('#include "sell.h"\n'
                'extern "C" int pad(const int *i, const int *o, const int *r, long long s, int w)'
                ' { return gb300::sell_pad_index(i, o, r, s, w); }\n')
    r = subprocess.run([cxx, "-std=c++17", "-shared", "-fPIC", "-I" + CUDA, "-I" + os.path.join(
        ROOT, "opensubdiv_gb300", "csrc"), src, "-o", lib], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(lib).pad


@pytest.mark.parametrize("n,empty", [(1, 0.0), (1, 1.0), (31, 0.5), (33, 0.9), (256, 0.97),
                                     (257, 0.5), (1000, 0.8), (3000, 0.99)])
def test_slots_of_empty_stencils(rule, n, empty):
    rng = np.random.default_rng(n)
    sizes = np.where(rng.random(n) < empty, 0, rng.integers(1, 20, n)).astype(np.int32)
    offsets = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int32)
    indices = rng.integers(100, 5000, max(1, int(sizes.sum()))).astype(np.int32)
    slices = -(-n // 32)
    # positions: sorted by size, largest first, within windows of 256; none behind the last stencil
    row = np.full(slices * 32, -1, np.int32)
    for w in range(0, n, 256):
        ids = np.arange(w, min(w + 256, n))
        row[w:w + len(ids)] = ids[np.argsort(-sizes[ids], kind="stable")]
    ptr = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_int))  # noqa: E731
    for s in range(slices):
        ids = [i for i in row[32 * s:32 * s + 32] if i >= 0]
        width = max(int(sizes[i]) for i in ids)
        got = rule(ptr(indices), ptr(offsets), ptr(row), ctypes.c_longlong(s), width)
        read = {int(x) for i in ids for x in indices[offsets[i]:offsets[i] + sizes[i]]}
        assert got in read if width else got == 0


def test_the_build_uses_it():
    text = open(os.path.join(ROOT, "opensubdiv_gb300", "csrc", "sell_build.cu")).read()
    assert "n > 0 ? 0 : sell_pad_index(indices, offsets, row, sl, width)" in text
    assert "idx[slot] = on ? indices[o + j] : pad;" in text
