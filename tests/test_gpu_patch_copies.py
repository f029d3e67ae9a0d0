"""The copies of a Loop table's rows that EvalPatches makes of many points (a quad per row, a quad per
patch index), and FindPatches of tables above and below the size from which handles are computed and
records written through shared memory: at the sizes where that changes and around a warp, packed and
strided outputs, against the oracle at the accuracy gate of tests/gpu_util.py."""
import os

import numpy as np
import pytest

import oracle
from gpu_util import bbox_diag_rows, dev, gate, host, torch_cuda

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


def _instances(name, copies):
    from opensubdiv_gb300 import workloads
    with np.load(os.path.join(GOLDEN, name + ".npz")) as f:
        z = {k: f[k] for k in f.files}
    if "num_ptex" not in z:
        z["num_ptex"] = z["ptex_offsets"][-1]
    return workloads.instanced_patch_table(z, copies)


def _queries(n, ptex, tri, seed):
    rng = np.random.default_rng(seed)
    face = rng.integers(-1, ptex + 1, n).astype(np.int32)
    u, v = rng.random(n, np.float32), rng.random(n, np.float32)
    if tri:
        fold = u + v > 1.0
        u[fold], v[fold] = 1.0 - u[fold], 1.0 - v[fold]
    return face, u, v


# 2358 rows per copy: a quad per row below 32768 rows, with derivatives a quad per index above,
# unless there are more indices than points (25 copies: 267 k)
@pytest.mark.gpu
@pytest.mark.parametrize("copies,points,stride,out_stride,outputs", [
    (1, (1 << 18) - 1, 3, 3, 6), (1, 1 << 18, 3, 3, 1), (1, (1 << 18) + 33, 5, 4, 6),
    (13, 1 << 18, 3, 3, 3), (4, (3 << 16) - 1, 3, 3, 3), (4, 3 << 16, 3, 3, 3), (14, 3 << 16, 3, 3, 6),
    (14, 1 << 18, 3, 3, 3), (14, (1 << 18) + 1, 4, 3, 6),
    (15, (1 << 18) + 31, 3, 5, 6), (15, 1 << 18, 3, 3, 1), (25, 1 << 18, 3, 3, 3)])
def test_copied_rows(copies, points, stride, out_stride, outputs):
    torch = torch_cuda()
    from opensubdiv_gb300.evaluator import (BufferDescriptor as BD, GB300Evaluator as Ev,
                                            GB300PatchTable)
    arrays, indices, params, src, ptex, tri = _instances("icosphere2_patches_L3", copies)
    xyz = src.reshape(-1, 3)
    rows = np.full((len(xyz), stride), np.nan, np.float32)  # what a wider row holds does not matter
    rows[:, :3] = xyz
    t = GB300PatchTable.Create(arrays, indices, params, tri)
    face, u, v = _queries(points, ptex, tri, points)
    coords = torch.zeros((points, 5), dtype=torch.int32, device="cuda")
    t.FindPatches(points, dev(face), dev(u), dev(v), coords)
    out = [torch.full((points, out_stride), 7.0, device="cuda") for _ in range(outputs)]
    d, kw = BD(0, 3, out_stride), {}
    for k, name in enumerate(("du", "dv", "duu", "duv", "dvv")[:outputs - 1]):
        kw[name], kw[name + "Desc"] = out[k + 1], d
    assert Ev.EvalPatchesTable(dev(rows.ravel()), BD(0, 3, stride), out[0], d, points, coords, t,
                               **kw)
    Ev.Synchronize()
    c = host(coords)
    hit = c[:, 0] >= 0
    assert 0 < (~hit).sum() < points // 3
    ref = []
    for fp64 in (False, True):
        o = [np.zeros(hit.sum() * 3, np.float64 if fp64 else np.float32) for _ in range(6)]
        oracle.eval_patches(src, (0, 3, 3), o, [(0, 3, 3)] * 6, np.ascontiguousarray(c[hit]),
                            arrays, indices, params, threads=8, fp64=fp64)
        ref.append(o)
    diag = bbox_diag_rows(src, 3)
    for k in range(outputs):
        got = host(out[k])
        assert (got[:, 3:] == 7.0).all() and (got[~hit][:, :3] == 0.0).all()
        gate("copied rows", k, got[hit][:, :3].ravel(), ref[0][k], ref[1][k], diag)


@pytest.mark.gpu
@pytest.mark.parametrize("table,copies", [("torus32x16_patches_L4", 2), ("torus32x16_patches_L4", 3),
                                          ("icosphere2_patches_L3", 19),
                                          ("icosphere2_patches_L3", 20)])
def test_records_of_both_kinds(table, copies):
    """12,214 and 18,321, 16,340 and 17,200 patches."""
    torch = torch_cuda()
    from opensubdiv_gb300.evaluator import GB300PatchTable
    arrays, indices, params, _, ptex, tri = _instances(table, copies)
    assert (len(params) < 1 << 14) == (copies in (2, 19))
    t = GB300PatchTable.Create(arrays, indices, params, tri)
    m = oracle.PatchMap(arrays, params, tri)
    for n in (1, 31, 32, 33, 255, 257, 70001):
        face, u, v = _queries(n, ptex, tri, n)
        out = torch.full((n + 7, 5), -5, dtype=torch.int32, device="cuda")
        t.FindPatches(n, dev(face), dev(u), dev(v), out)
        torch.cuda.synchronize()
        got = host(out)
        assert (got[n:] == -5).all()
        assert np.array_equal(got[:n, :3], np.asarray(m.find(face, u, v))[:, :3])
        assert np.array_equal(got[:n, 3], u.view(np.int32))
        assert np.array_equal(got[:n, 4], v.view(np.int32))
