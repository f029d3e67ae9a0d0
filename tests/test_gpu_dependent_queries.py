"""Queries, patch coords, refined points and padded copies that are written again while the kernels
that read them are already resident: stencils -> FindPatches -> EvalPatches, and Generate -> Evaluate,
each step over the same buffers with other contents, give the bits of the same calls with a
synchronisation after each.

Loop tables of more points than control rows and patch indices evaluate from a copy in scratch memory
(a row per control point for P alone, a row per patch index with derivatives), which the next step's
copy overwrites; Catmull-Clark tables read the source itself.
"""
import os

import numpy as np
import pytest

from gpu_util import dev, torch_cuda

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
STEPS = 6


def _tables(name):
    """The patch table, and a stencil table that writes all rows the patches read from the cage."""
    from opensubdiv_gb300.evaluator import GB300PatchTable, GB300StencilTable
    z = np.load(os.path.join(GOLDEN, name + ".npz"))
    t = GB300PatchTable.Create(z["arrays"], z["patch_indices"], z["params"],
                               triangular=bool(z["triangular"]))
    n = len(z["positions"])
    sizes = np.concatenate([np.ones(n, np.int32), z["ps_sizes"]]).astype(np.int32)
    offsets = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int32)
    st = GB300StencilTable.Create(sizes, offsets,
                                  np.concatenate([np.arange(n), z["ps_indices"]]).astype(np.int32),
                                  np.concatenate([np.ones(n), z["ps_weights"]]).astype(np.float32))
    return z, t, st, len(sizes)


def _run(steps, sync):
    from opensubdiv_gb300.evaluator import GB300Evaluator as Ev
    for calls in steps:
        for call in calls:
            call()
            if sync:
                Ev.Synchronize()
    Ev.Synchronize()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["icosphere2_patches_L3", "torus32x16_patches_L4"])
@pytest.mark.parametrize("points", [3000, 70001])
@pytest.mark.parametrize("outputs", [1, 3, 6])
def test_stencils_find_and_evaluate(name, points, outputs):
    torch = torch_cuda()
    from opensubdiv_gb300.evaluator import BufferDescriptor as BD, GB300Evaluator as Ev
    z, table, refine, rows = _tables(name)
    rng = np.random.default_rng(points + outputs)
    d = BD(0, 3, 3)
    src = torch.zeros(rows * 3, device="cuda")
    records = torch.zeros(points * 5, dtype=torch.int32, device="cuda")
    outs = torch.zeros(STEPS, 6, points * 3, device="cuda")
    steps = []
    for k in range(STEPS):
        cage = dev((z["positions"] * rng.uniform(0.5, 2.0, (1, 3))).astype(np.float32).ravel())
        q = rng.integers(0, len(z["q_face"]), points)
        f, u, v = (dev(z[x][q]) for x in ("q_face", "q_u", "q_v"))
        kw = {}
        for i, x in enumerate(("du", "dv", "duu", "duv", "dvv")[:outputs - 1]):
            kw[x], kw[x + "Desc"] = outs[k, i + 1], d
        steps.append([
            lambda cage=cage: Ev.EvalStencilsTable(cage, d, src, d, refine),
            lambda f=f, u=u, v=v: table.FindPatches(points, f, u, v, records),
            lambda k=k, kw=kw: Ev.EvalPatchesTable(src, d, outs[k, 0], d, points, records, table,
                                                   **kw)])
    _run(steps, True)
    want = outs.clone()
    assert want[:, :outputs].abs().amax(dim=2).min() > 0
    for _ in range(4):
        outs.zero_()
        records.zero_()
        src.zero_()
        _run(steps, False)
        assert torch.equal(outs, want)


@pytest.mark.gpu
@pytest.mark.parametrize("name,reg", [("icosphere2_patches_L3", 3), ("torus32x16_patches_L4", 4)])
def test_generate_and_evaluate(name, reg):
    torch = torch_cuda()
    from opensubdiv_gb300 import bfr
    from opensubdiv_gb300.evaluator import BufferDescriptor as BD, GB300Evaluator as Ev
    z, table, refine, rows = _tables(name)
    rng = np.random.default_rng(reg)
    d = BD(0, 3, 3)
    src = torch.zeros(rows * 3, device="cuda")
    meshes = [bfr.MeshTessellation(reg, z["verts_per_face"],
                                   rates=rng.integers(1, 9, len(z["verts_per_face"])))
              for _ in range(STEPS)]
    most = max(m.num_coords for m in meshes)
    coords = torch.zeros(most, 2, device="cuda")
    facets = torch.zeros(max(m.num_facets for m in meshes), 3, dtype=torch.int32, device="cuda")
    records = torch.zeros(most, 5, dtype=torch.int32, device="cuda")
    outs = [[torch.zeros(m.num_coords, 3, device="cuda") for _ in range(3)] for m in meshes]
    steps = []
    for m, o in zip(meshes, outs):
        cage = dev((z["positions"] * rng.uniform(0.5, 2.0, (1, 3))).astype(np.float32).ravel())
        steps.append([
            lambda cage=cage: Ev.EvalStencilsTable(cage, d, src, d, refine),
            lambda m=m: m.Generate(coords, facets, table=table, patch_coords=records),
            lambda m=m, o=o: m.Evaluate(src, d, table, records, derivatives=1, outputs=o)])
    _run(steps, True)
    want = [[x.clone() for x in o] for o in outs]
    assert min(float(x.abs().max()) for o in want for x in o) > 0
    for _ in range(4):
        for o in outs:
            for x in o:
                x.zero_()
        for b in (coords, facets, records, src):
            b.zero_()
        _run(steps, False)
        assert all(torch.equal(a, b) for x, y in zip(outs, want) for a, b in zip(x, y))
