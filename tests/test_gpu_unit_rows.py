"""The unit layout of a regular table (slices whose units share their weights) at output rows with gaps
and at its larger units, against the oracle: rows of 1 to 15 floats inside wider 16-byte aligned rows,
written row by row or collected, below and above the size at which that changes, in single calls and
in a batch; and a table large enough for units of 16 stencils, with groups around that number, weights
that slices share and weights that they do not, and lists of up to 40 entries.

Tolerance: the rounding bound of two summation orders of the same entries, (2 n + 2) 2^-24 sum |w x|.
"""
import numpy as np
import pytest

import oracle
from gpu_util import dev, host, torch_cuda
from test_gpu_unit_layout import NCV, _check


def _regular(n, k=7, group=16, seed=3):
    """n stencils, every `group` of them over k control vertices of their own, the same weights."""
    rng = np.random.default_rng(seed)
    first = rng.integers(0, NCV - k, n // group)
    idx = (np.repeat(first, group)[:, None] + np.arange(k)).astype(np.int32).ravel()
    w = np.tile(rng.uniform(-0.2, 1.0, (group, k)).astype(np.float32), (n // group, 1)).ravel()
    return np.full(n, k, np.int32), (np.arange(n) * k).astype(np.int32), idx, w


@pytest.fixture(scope="module")
def regular():
    torch_cuda()
    from opensubdiv_gb300.evaluator import GB300StencilTable
    out = []
    for n in (1 << 19, 3 << 19):
        t = _regular(n)
        out.append((n, t, GB300StencilTable.Create(*t)))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("length,stride,out_stride", [
    (1, 4, 4), (2, 4, 4), (3, 4, 4), (3, 4, 8), (4, 4, 4), (4, 4, 8), (5, 8, 8), (6, 8, 8), (7, 8, 8),
    (7, 8, 12), (8, 8, 12), (8, 8, 16), (9, 12, 12), (10, 12, 12), (11, 12, 12), (12, 12, 16),
    (13, 16, 16), (15, 16, 16)])
def test_rows_with_gaps(regular, length, stride, out_stride):
    """1.5 M stencils: rows of 12 and 16 floats are above the size from which they are collected."""
    torch = torch_cuda()
    from opensubdiv_gb300.evaluator import BufferDescriptor as BD, GB300Evaluator as Ev
    from opensubdiv_gb300.evaluator import GB300StencilBatch
    rng = np.random.default_rng(length)
    jobs, plain = [], []
    for n, t, table in regular:
        src = rng.uniform(-1, 1, NCV * stride).astype(np.float32)
        s, sd, dd = dev(src), BD(0, length, stride), BD(0, length, out_stride)
        out = torch.zeros(n * out_stride, device="cuda")
        assert Ev.EvalStencilsTable(s, sd, out, dd, table)
        Ev.Synchronize()
        _check(host(out).reshape(-1), src, (0, length, stride), (0, length, out_stride), n, t)
        plain.append(out)
        jobs.append((table, s, sd, torch.zeros_like(out), dd))
    for run in ("Eval", "EvalGraph"):
        for j in jobs:
            j[3].zero_()
        batch = GB300StencilBatch(jobs)
        getattr(batch, run)()
        torch.cuda.synchronize()
        assert batch.GetDeviceStatus() == 0
        for j, p in zip(jobs, plain):
            assert torch.equal(j[3], p)


@pytest.fixture(scope="module")
def large():
    """4.3 M stencils in random order: copies of a base whose groups have 9 to 40 stencils, a third
    of the copies with weights of their own."""
    torch_cuda()
    from opensubdiv_gb300.evaluator import GB300StencilTable
    rng = np.random.default_rng(16)
    sizes, idx, w = [], [], []
    lists = [0, 1, 4, 5, 9, 15, 16, 16, 17, 40]
    while sum(len(s) for s in sizes) < 66000:
        k = int(rng.choice(lists))
        m = int(rng.choice([9, 15, 16, 17, 25, 32, 33, 40]))
        ids = np.sort(rng.integers(0, 300) + rng.choice(2 * k + 1, k, replace=False))
        ws = np.random.default_rng(100 * k + m).uniform(-0.2, 1.0, (m, k))
        sizes.append(np.full(m, k, np.int32))
        idx.append(np.tile(ids, m))
        w.append(ws.ravel())
    sizes, idx, w = (np.concatenate(x) for x in (sizes, idx, w))
    copies = 65
    n = len(sizes) * copies
    assert n >= 4 << 20
    I = np.concatenate([idx + 70 * c for c in range(copies)]).astype(np.int32)
    W = np.concatenate([w * (rng.uniform(0.5, 1.0, len(w)) if c % 3 == 0 else 1.0)
                        for c in range(copies)]).astype(np.float32)
    assert I.max() < NCV
    S = np.tile(sizes, copies)
    first = np.concatenate([[0], np.cumsum(S)[:-1]])
    order = np.concatenate([rng.permutation(len(sizes)) + c * len(sizes) for c in range(copies)])
    sizes = S[order]
    offsets = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int32)
    at = np.repeat(first[order] - offsets, sizes) + np.arange(len(I))
    t = (sizes, offsets, I[at], W[at])
    return n, t, GB300StencilTable.Create(*t)


@pytest.mark.gpu
@pytest.mark.parametrize("sd,dd", [((0, 4, 4), (0, 4, 4)), ((0, 8, 8), (0, 8, 8)),
                                   ((4, 8, 16), (4, 8, 12)), ((0, 5, 8), (0, 5, 5)),
                                   ((0, 12, 12), (0, 12, 12)), ((0, 16, 16), (0, 16, 16))])
def test_units_of_sixteen(large, sd, dd):
    torch = torch_cuda()
    from opensubdiv_gb300.evaluator import BufferDescriptor as BD, GB300Evaluator as Ev
    from opensubdiv_gb300.evaluator import GB300StencilBatch
    n, t, table = large
    src = np.random.default_rng(sd[1]).uniform(-1, 1, NCV * sd[2] + sd[0]).astype(np.float32)
    s = dev(src)
    out = torch.zeros(n * dd[2] + dd[0], device="cuda")
    assert Ev.EvalStencilsTable(s, BD(*sd), out, BD(*dd), table)
    Ev.Synchronize()
    _check(host(out).reshape(-1), src, sd, dd, n, t)
    again = torch.zeros_like(out)
    batch = GB300StencilBatch([(table, s, BD(*sd), again, BD(*dd))])
    batch.EvalGraph()
    torch.cuda.synchronize()
    assert batch.GetDeviceStatus() == 0 and torch.equal(again, out)
