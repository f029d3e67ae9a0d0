"""The rule for the unit layout's output rows, over lengths, strides, alignments and sizes, on the CPU:
rows are written by quads only where they are 16-byte aligned, tables below the layout's size of a
single call stay with the sliced layout, and so do irregular tables' narrow and ragged rows."""
import os
import shutil
import subprocess

import numpy as np
import pytest

CPP = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp")


def test_rule(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path / "unit_rows")
    cmd = [nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17",
           "--expt-relaxed-constexpr", os.path.join(CPP, "unit_rows.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0
    n, regular, length, stride, offset, batch, way = np.array(
        [line.split() for line in r.stdout.splitlines()], np.int64).T
    aligned = (stride % 4 == 0) & (offset % 4 == 0)
    assert not (way[~aligned] == 1).any()
    assert not way[(n < 262144) & (batch == 0)].any()
    single, few = batch == 0, n * stride * 4 < 64 << 20
    # unaligned rows of a single call: large regular tables only
    assert ((way[single & ~aligned] == 2) ==
            ((n >= 3 << 19) & (regular == 1))[single & ~aligned]).all()
    # whole quads of 8 and more floats, and rows of 16 and more, always
    whole = aligned & (length % 4 == 0) & (length == stride) & (length > 4)
    assert (way[(whole | (aligned & (length >= 16))) & ((n >= 262144) | (batch == 1))] == 1).all()
    # an irregular table's rows narrower than a quad, and tails of 2 and 3 floats up to 12, never
    ragged = aligned & (regular == 0) & ((length < 4) | ((length % 4 > 1) & (length < 8)))
    assert not way[ragged].any()
    # nor its rows with gaps once they outgrow the L2
    gap = aligned & (regular == 0) & (length <= 12) & (stride > length) & (stride % 8 != 0)
    assert not way[gap & (n * stride * 4 > 130 << 20)].any()
    # regular tables: a few megabytes of rows row by row, a tail beyond that collected
    some = aligned & (regular == 1) & single & (n >= 262144) & (length > 4)
    assert (way[some & few & (stride - length < 4)] == 1).all()
    tail = some & (length % 4 != 0) & (length < 12) & (stride - length < 4)
    assert (way[tail & (n * stride * 4 > 66 << 20)] == 2).all()
