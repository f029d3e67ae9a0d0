"""A batch whose jobs need all five kinds of kernel (general, narrow, wide, unit rows, unit rows
collected): the bits of its plain calls, by Eval and by the graph, whose parts are branches, over
sources written again between replays, before and after tuning; and what the tuner times, on the
sources."""
import os
import re

import numpy as np
import pytest

from gpu_util import host, torch_cuda

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "opensubdiv_gb300", "csrc")


def test_the_tuner_times_both_ways():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "stencils_batch.cu")).read())
    body = text[text.index("int GB300StencilBatchTune("):]
    timed = body[body.index("cudaEventRecord(e0"):body.index("cudaEventRecord(e1")]
    assert "launch_batch(b, s)" in timed and "launch_graph(b, s)" in timed
    before = body[body.index("upload_plan(b, s)"):body.index("cudaEventRecord(e0")]
    assert before.index("drop_graph") < before.index("launch_graph(b, s)")  # of this configuration
    assert body.index("drop_graph", body.index("done:")) < body.index("b->cfg = best")


@pytest.mark.gpu
@pytest.mark.parametrize("dynamic_order", [False, True])
def test_all_parts(dynamic_order):
    torch = torch_cuda()
    from opensubdiv_gb300.evaluator import BufferDescriptor as BD, GB300Evaluator as Ev
    from opensubdiv_gb300.evaluator import GB300StencilBatch, GB300StencilTable
    from test_gpu_unit_layout import NCV, _check, _table
    rng = np.random.default_rng(31)
    jobs, plain, host_of = [], [], []
    # stencils, length, source stride, output stride
    kinds = [(9001, 7, 8, 8), (70003, 5, 5, 5), (12007, 3, 4, 4), (8009, 12, 12, 12),
             (90001, 8, 8, 8), (66001, 12, 12, 12), (5003, 16, 16, 16), (300, 3, 3, 3),
             (80021, 11, 12, 11)]
    if dynamic_order:
        kinds = kinds[::-1]
    for n, length, stride, out_stride in kinds:
        t = _table(n, n + length)
        s = torch.zeros(NCV * stride, device="cuda")
        jobs.append((GB300StencilTable.Create(*t), s, BD(0, length, stride),
                     torch.zeros(n * out_stride, device="cuda"), BD(0, length, out_stride)))
        plain.append(torch.zeros(n * out_stride, device="cuda"))
        host_of.append((n, t))
    batch = GB300StencilBatch(jobs)

    def frame(run):
        srcs = []
        for j in jobs:
            srcs.append(rng.uniform(-1, 1, j[1].numel()).astype(np.float32))
            j[1].copy_(torch.from_numpy(srcs[-1]))
            j[3].zero_()
        run()
        for (table, s, sd, _, dd), p in zip(jobs, plain):
            assert Ev.EvalStencilsTable(s, sd, p, dd, table)
        torch.cuda.synchronize()
        assert batch.GetDeviceStatus() == 0
        for j, p in zip(jobs, plain):
            assert torch.equal(j[3], p)
        return srcs

    for run in (batch.Eval, batch.EvalGraph, batch.EvalGraph):
        srcs = frame(run)
    for j, src, (n, t), (_, length, stride, out_stride) in zip(jobs, srcs, host_of, kinds):
        _check(host(j[3]).reshape(-1), src, (0, length, stride), (0, length, out_stride), n, t)
    batch.Tune(iterations=2)
    for run in (batch.EvalGraph, batch.Eval, batch.EvalGraph):
        frame(run)
