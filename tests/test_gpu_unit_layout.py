"""Large stencil tables evaluate aligned rows through their unit layout (stencils with the same
control vertices evaluated together, weights that a whole slice shares held once): against the
oracle at the edges of that layout.

Covered: lists of 0, 1, 3-5, 15, 16 (held in registers), 17, 40 (16 at a time) and 365 entries
(longer than the staging ring), groups of 1 to 70 stencils (units of 1 to 8 or 16), weights that
slices share and weights that they do not, stencils in random table order, partial last slices, rows
of 3 to 33 floats inside wider strides, a control point at infinity, and the same table through a
batch.  Tolerance: the rounding bound of two summation orders of the same entries.
"""
import numpy as np
import pytest

import oracle
from gpu_util import dev, host, torch_cuda

NCV = 5000


def _table(n, seed):
    """n stencils in groups of equal lists, most groups with weights of a pool, shuffled."""
    rng = np.random.default_rng(seed)
    pool = {}
    sizes, idx, w = [], [], []
    while len(sizes) < n:
        k = int(rng.choice([0, 1, 3, 4, 5, 9, 12, 15, 16, 16, 16, 17, 40, 365],
                           p=[.02, .05, .05, .08, .08, .1, .1, .1, .1, .1, .1, .08, .037, .003]))
        m = min(int(rng.choice([1, 2, 8, 9, 16, 25, 70])) if k <= 40 else 1, n - len(sizes))
        lo = int(rng.integers(0, NCV - 2 * k - 2))
        ids = np.sort(lo + rng.choice(2 * k + 1, k, replace=False)).astype(np.int32)
        if rng.random() < 0.7:
            if (k, m) not in pool:
                pool[k, m] = rng.uniform(-0.2, 1.0, (m, k)).astype(np.float32)
            ws = pool[k, m]
        else:
            ws = rng.uniform(-0.2, 1.0, (m, k)).astype(np.float32)
        for i in range(m):
            sizes.append(k)
            idx.append(ids)
            w.append(ws[i])
    order = rng.permutation(n)
    sizes = np.array(sizes, np.int32)[order]
    offsets = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int32)
    return (sizes, offsets, np.concatenate([idx[i] for i in order]),
            np.concatenate([w[i] for i in order]))


@pytest.fixture(scope="module")
def tables():
    torch_cuda()
    from opensubdiv_gb300.evaluator import GB300StencilTable
    out = []
    for n in (262144, 300007):
        t = _table(n, n)
        out.append((n, t, GB300StencilTable.Create(*t)))
    return out


def _check(got, src, sd, dd, n, t):
    sizes, offsets, idx, w = t
    ref = np.zeros(n * dd[2] + dd[0], np.float32)
    oracle.eval_stencils(src, sd, [ref], [dd], sizes, offsets, idx, [w], threads=8)
    # both orders of summation are within (size - 1) u sum |w x| of the exact sum
    a = oracle.stencil_abs_scale(src, sd, sizes, offsets, idx, w).reshape(n, -1)
    bound = (2.0 * np.maximum(sizes, 1)[:, None] + 2.0) * 2.0 ** -24 * a + 1e-7
    off, ln, st = dd
    g = got[off: off + n * st].reshape(n, st).copy()
    r = ref[off: off + n * st].reshape(n, st)[:, :ln]
    ok = np.isfinite(r)
    assert np.array_equal(ok, np.isfinite(g[:, :ln]))
    assert (np.abs(g[:, :ln][ok].astype(np.float64) - r[ok]) <= bound[ok]).all()
    g[:, :ln] = 0.0
    assert not g.any()  # elements outside the rows stay untouched


@pytest.mark.gpu
@pytest.mark.parametrize("sd,dd", [((0, 4, 4), (0, 4, 4)), ((4, 3, 8), (0, 3, 4)),
                                   ((0, 8, 8), (0, 8, 8)), ((0, 5, 8), (4, 5, 12)),
                                   ((0, 12, 12), (0, 12, 12)), ((0, 11, 12), (0, 11, 12)),
                                   ((0, 16, 16), (0, 16, 16)), ((0, 33, 36), (0, 33, 36)),
                                   ((0, 8, 9), (0, 8, 8))])
def test_rows_and_sizes(tables, sd, dd):
    torch = torch_cuda()
    from opensubdiv_gb300.evaluator import BufferDescriptor as BD, GB300Evaluator as Ev
    rng = np.random.default_rng(sd[1])
    for n, t, table in tables:
        src = rng.uniform(-1, 1, NCV * sd[2] + sd[0]).astype(np.float32)
        out = torch.zeros(n * dd[2] + dd[0], device="cuda")
        assert Ev.EvalStencilsTable(dev(src), BD(*sd), out, BD(*dd), table)
        Ev.Synchronize()
        _check(host(out).reshape(-1), src, sd, dd, n, t)


@pytest.mark.gpu
def test_infinite_control_point_and_batch(tables):
    """Only the stencils that read a control point at infinity are not finite; a batch of the two
    tables (and one of another width) writes the bits of the plain calls."""
    torch = torch_cuda()
    from opensubdiv_gb300.evaluator import BufferDescriptor as BD, GB300Evaluator as Ev
    from opensubdiv_gb300.evaluator import GB300StencilBatch
    rng = np.random.default_rng(5)
    jobs, plain = [], []
    for k, (n, t, table) in enumerate(tables + tables[:1]):
        L = (8, 12, 7)[k]
        src = rng.uniform(-1, 1, NCV * L).astype(np.float32)
        src[0] = np.inf  # control point 0, which the padding of the layout also names
        src[7 * L + 1] = np.nan
        d, s = BD(0, L, L), dev(src)
        out = torch.zeros(n * L, device="cuda")
        assert Ev.EvalStencilsTable(s, d, out, d, table)
        Ev.Synchronize()
        _check(host(out).reshape(-1), src, (0, L, L), (0, L, L), n, t)
        plain.append(out)
        jobs.append((table, s, d, torch.zeros_like(out), d))
    batch = GB300StencilBatch(jobs)
    for run in (batch.Eval, batch.EvalGraph):
        for j in jobs:
            j[3].zero_()
        run()
        torch.cuda.synchronize()
        for j, p in zip(jobs, plain):
            assert torch.equal(torch.nan_to_num(j[3]), torch.nan_to_num(p))
    assert batch.GetDeviceStatus() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("length,stride,out_stride", [(3, 3, 3), (5, 5, 5), (3, 4, 5), (7, 8, 7),
                                                      (11, 11, 11), (20, 20, 21)])
def test_unaligned_output_rows(length, stride, out_stride):
    """Output rows that no vector store takes (collected before they are written): a batch of tables
    above and below the layout's size, and a single call on a regular table large enough for it."""
    torch = torch_cuda()
    from opensubdiv_gb300.evaluator import BufferDescriptor as BD, GB300Evaluator as Ev
    from opensubdiv_gb300.evaluator import GB300StencilBatch, GB300StencilTable
    rng = np.random.default_rng(length)
    jobs, want = [], []
    for n in (65535, 65536, 100003):
        t = _table(n, n + length)
        src = rng.uniform(-1, 1, NCV * stride).astype(np.float32)
        out = torch.zeros(n * out_stride, device="cuda")
        jobs.append((GB300StencilTable.Create(*t), dev(src), BD(0, length, stride), out,
                     BD(0, length, out_stride)))
        want.append((src, (0, length, stride), (0, length, out_stride), n, t))
    GB300StencilBatch(jobs).Eval()
    torch.cuda.synchronize()
    for j, w in zip(jobs, want):
        _check(host(j[3]).reshape(-1), *w)
    # 98304 groups of 16 stencils with the same weights: 1.5 M stencils
    n, k = 3 << 19, 7
    first = rng.integers(0, NCV - k, n // 16)
    idx = (np.repeat(first, 16)[:, None] + np.arange(k)).astype(np.int32).ravel()
    w = np.tile(rng.uniform(-0.2, 1.0, (16, k)).astype(np.float32), (n // 16, 1)).ravel()
    t = (np.full(n, k, np.int32), (np.arange(n) * k).astype(np.int32), idx, w)
    table = GB300StencilTable.Create(*t)
    src = rng.uniform(-1, 1, NCV * stride).astype(np.float32)
    out = torch.zeros(n * out_stride, device="cuda")
    assert Ev.EvalStencilsTable(dev(src), BD(0, length, stride), out, BD(0, length, out_stride),
                                table)
    Ev.Synchronize()
    _check(host(out).reshape(-1), src, (0, length, stride), (0, length, out_stride), n, t)
