"""EvalPatches over the source and output layouts that choose a kernel: Loop tables with more points
than source rows (a copy padded to quads), or than patch indices (a copy of a row per index), rows of whole quads, packed outputs (written through shared
memory, whole sectors at a time) and outputs inside wider rows, at point counts around a warp and
around the padded copy's threshold.  Accuracy gate of tests/gpu_util.py (1e-5 x the bounding-box
diagonal against the oracle, second derivatives against its FP64 form)."""
import os

import numpy as np
import pytest

import oracle
from gpu_util import bbox_diag_rows, dev, gate, host, smooth_primvars, torch_cuda

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


@pytest.mark.gpu
@pytest.mark.parametrize("table", ["icosphere2_patches_L3", "trigrid6_patches_L3",
                                   "torus32x16_patches_L4"])
@pytest.mark.parametrize("points,length,stride,out_stride,outputs", [
    (1, 3, 3, 3, 6), (31, 4, 4, 4, 3), (33, 4, 8, 4, 6), (257, 8, 8, 8, 6), (65535, 3, 3, 3, 3),
    (65536, 3, 3, 3, 6), (65569, 3, 3, 4, 6), (65537, 3, 4, 3, 1), (66001, 3, 5, 3, 3)])
def test_rows_and_counts(table, points, length, stride, out_stride, outputs, more=0):
    torch = torch_cuda()
    from opensubdiv_gb300.evaluator import (BufferDescriptor as BD, GB300Evaluator as Ev,
                                            GB300PatchTable)
    z = np.load(os.path.join(GOLDEN, table + ".npz"))
    xyz = z["src"].reshape(-1, 3)
    rows = np.zeros((len(xyz), stride), np.float32)
    rows[:, :length] = (smooth_primvars(xyz)[:, :length] if length > 3 else xyz)
    rows[:, length:] = np.nan  # what a wider row holds must not reach the result
    coords = z["coords"][np.arange(points) % len(z["coords"])]
    indices = np.concatenate([z["patch_indices"], np.zeros(more, np.int32)])
    t = GB300PatchTable.Create(z["arrays"], indices, z["params"],
                               triangular=bool(z["triangular"]))
    out = [torch.full((points * out_stride,), 7.0, device="cuda") for _ in range(outputs)]
    d, kw = BD(0, length, out_stride), {}
    for k, name in enumerate(("du", "dv", "duu", "duv", "dvv")[:outputs - 1]):
        kw[name], kw[name + "Desc"] = out[k + 1], d
    assert Ev.EvalPatchesTable(dev(rows.ravel()), BD(0, length, stride), out[0], d, points,
                               dev(coords), t, **kw)
    Ev.Synchronize()
    ref = []
    for fp64 in (False, True):
        o = [np.zeros(points * length, np.float64 if fp64 else np.float32) for _ in range(6)]
        oracle.eval_patches(rows[:, :length].copy().ravel(), (0, length, length), o,
                            [(0, length, length)] * 6, coords, z["arrays"], z["patch_indices"],
                            z["params"], threads=8, fp64=fp64)
        ref.append(o)
    diag = bbox_diag_rows(rows[:, :length].copy(), length)
    for k in range(outputs):
        got = host(out[k]).reshape(points, out_stride)
        gate(f"{table} rows", k, got[:, :length].ravel(), ref[0][k], ref[1][k], diag)
        assert (got[:, length:] == 7.0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("outputs", [1, 3, 6])
def test_more_indices_than_points(outputs):
    """More points than source rows, but not than patch indices (the last ones unused)."""
    test_rows_and_counts("icosphere2_patches_L3", 65536, 3, 3, 3, outputs, more=65536)
