"""When a table gets its unit layout: with the table from the size on at which single calls may take
it, else from the first batch, once, also when batches of several threads are made at the same time."""
import os
import re
import threading

import numpy as np
import pytest

from gpu_util import dev, torch_cuda

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "opensubdiv_gb300", "csrc")


def test_single_calls_read_no_layout_that_a_batch_may_build():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "objects.cu")).read())
    body = text[text.index("int table_eval(const GB300StencilTable *t, const float *src, float *const *dIn"):]
    body = body[:body.index("eval_stencils_units")]
    assert body.index("t->numStencils >= kUnitCall") < body.index("t->unit")
    body = text[text.index("int stencil_table_units("):]
    body = body[:body.index("\n}")]
    assert "t->numStencils < kUnitCall" in body and body.index("lock") < body.index("build_unit")


@pytest.mark.gpu
def test_built_once_and_when_needed():
    torch = torch_cuda()
    from opensubdiv_gb300 import _lib
    from opensubdiv_gb300.evaluator import BufferDescriptor as BD, GB300Evaluator as Ev
    from opensubdiv_gb300.evaluator import GB300StencilBatch, GB300StencilTable
    from test_gpu_unit_layout import NCV, _table
    d, rng = BD(0, 8, 8), np.random.default_rng(4)

    def launches(f):
        before = _lib.launch_count()
        r = f()
        return r, _lib.launch_count() - before

    made = {n: launches(lambda: GB300StencilTable.Create(*_table(n, n)))
            for n in (65535, 65537, 100003, 262144)}
    assert made[65535][1] == made[65537][1] == made[100003][1] < made[262144][1]
    src = dev(rng.uniform(-1, 1, NCV * 8).astype(np.float32))
    table = made[100003][0]
    plain = torch.zeros(100003 * 8, device="cuda")
    assert Ev.EvalStencilsTable(src, d, plain, d, table)

    def job():
        return table, src, d, torch.zeros(100003 * 8, device="cuda"), d

    one, n = launches(lambda: GB300StencilBatch([job()]))  # too few stencils: not built
    assert n == 0
    jobs = [[job(), job()] for _ in range(8)]
    batches, errors = [None] * 8, []

    def make(k):
        try:
            torch.cuda.set_device(0)
            batches[k] = GB300StencilBatch(jobs[k], stream=torch.cuda.Stream())
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    def all_at_once():
        threads = [threading.Thread(target=make, args=(k,)) for k in range(8)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()

    _, n = launches(all_at_once)
    assert not errors and n == made[262144][1] - made[65535][1]  # one build
    for b, js in zip(batches, jobs):
        b.EvalGraph()
        torch.cuda.synchronize()
        assert all(torch.equal(j[3], plain) for j in js) and b.GetDeviceStatus() == 0
