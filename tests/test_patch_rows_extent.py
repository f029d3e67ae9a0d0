"""Source rows that EvalPatches of a Loop table may read, on the CPU over a faked CUDA runtime (see
tests/cpp/patch_rows_extent.cu), and on the GPU over a buffer without the rows that no point needs."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from gpu_util import dev, torch_cuda

HERE = os.path.dirname(os.path.abspath(__file__))


def test_the_copy_stays_in_the_buffer(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path / "patch_rows_extent")
    cmd = [nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17",
           "--expt-relaxed-constexpr", "--cudart=none",
           os.path.join(HERE, "cpp", "patch_rows_extent.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("outputs,copies", [(1, 2), (6, 2), (6, 15)])
def test_rows_that_no_point_needs_may_be_missing(outputs, copies):
    """Instances of a Loop mesh, the points all in the first, whose rows are all that the buffer
    has: the bits of calls of fewer points, which read the rows of their patches only."""
    torch = torch_cuda()
    from opensubdiv_gb300 import workloads
    from opensubdiv_gb300.evaluator import (BufferDescriptor as BD, GB300Evaluator as Ev,
                                            GB300PatchTable, GB300VertexBuffer)
    with np.load(os.path.join(HERE, "golden", "icosphere2_patches_L3.npz")) as f:
        z = {k: f[k] for k in f.files}
    if "num_ptex" not in z:
        z["num_ptex"] = z["ptex_offsets"][-1]
    arrays, indices, params, _, ptex, tri = workloads.instanced_patch_table(z, copies)
    table = GB300PatchTable.Create(arrays, indices, params, tri)
    n = (1 << 18) + 33
    rng = np.random.default_rng(9)
    face = rng.integers(0, int(z["num_ptex"]), n).astype(np.int32)
    u, v = rng.random(n, np.float32), rng.random(n, np.float32)
    fold = u + v > 1.0
    u[fold], v[fold] = 1.0 - u[fold], 1.0 - v[fold]
    coords = torch.zeros((n, 5), dtype=torch.int32, device="cuda")
    table.FindPatches(n, dev(face), dev(u), dev(v), coords)
    assert (coords[:, 0] >= 0).all()
    rows = z["src"].astype(np.float32).reshape(-1, 3)
    buffer = GB300VertexBuffer.Create(3, rows.shape[0])
    buffer.UpdateData(rows, 0, rows.shape[0])
    d, got = BD(0, 3, 3), []
    for step in (n, 100000):
        out = [torch.zeros((n, 3), device="cuda") for _ in range(outputs)]
        for lo in range(0, n, step):
            m, kw = min(step, n - lo), {}
            for k, name in enumerate(("du", "dv", "duu", "duv", "dvv")[:outputs - 1]):
                kw[name], kw[name + "Desc"] = out[k + 1][lo:], d
            assert Ev.EvalPatchesTable(buffer, d, out[0][lo:], d, m, coords[lo:], table, **kw)
        torch.cuda.synchronize()
        got.append(out)
    for a, b in zip(*got):
        assert torch.equal(a, b) and a.abs().sum() > 0
