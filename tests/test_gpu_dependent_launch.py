"""Evaluators queued back to back, whose kernels may start while the one before still runs: each
reads what the one before writes, and overwrites what the one before that reads.

The chain of calls gives the bits of the same calls with a synchronisation after each, on a side
stream and replayed from a captured graph.  Tables: one that evaluates through the sliced layout,
one through the unit layout, and one whose unaligned source is copied to padded rows first.
"""
import numpy as np
import pytest

from gpu_util import dev, torch_cuda


def _table(n, ncv, k, groups, seed):
    """n stencils of k entries, `groups` of them alike in a row, over ncv points."""
    rng = np.random.default_rng(seed)
    first = np.repeat(rng.integers(0, ncv - k, -(-n // groups)), groups)[:n]
    idx = (first[:, None] + np.arange(k)).astype(np.int32).ravel()
    w = rng.uniform(0, 2.0 / k, n * k).astype(np.float32)
    return np.full(n, k, np.int32), (np.arange(n) * k).astype(np.int32), idx, w


@pytest.mark.gpu
@pytest.mark.parametrize("length,stride", [(3, 3), (4, 4), (8, 8), (5, 5)])
def test_chain_of_dependent_calls(length, stride):
    torch = torch_cuda()
    from opensubdiv_gb300.evaluator import BufferDescriptor as BD, GB300Evaluator as Ev
    from opensubdiv_gb300.evaluator import GB300StencilTable
    m = 1 << 18
    tables = [GB300StencilTable.Create(*_table(m, m, k, g, k + length))
              for k, g in ((3, 1), (5, 8), (9, 4))]  # 0.8 M, 1.3 M and 2.4 M entries
    d = BD(0, length, stride)
    start = dev(np.random.default_rng(length).uniform(-1, 1, m * stride).astype(np.float32))
    a, b = start.clone(), torch.zeros_like(start)

    def chain(sync, stream=None):
        x, y = a, b
        for step in range(8):
            assert Ev.EvalStencilsTable(x, d, y, d, tables[step % 3], stream=stream)
            if sync:
                Ev.Synchronize()
            x, y = y, x

    chain(True)
    want = [a.clone(), b.clone()]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            a.copy_(start)
            b.zero_()
            chain(False, side)
            got = [a.clone(), b.clone()]
            side.synchronize()
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        a.copy_(start)
        b.zero_()
        chain(False, side)
    for _ in range(2):
        a.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(a, want[0]) and torch.equal(b, want[1])
