"""Rows of at most 4 floats (xyz padded to quads, 4-wide primvars) with 1-6 outputs of a limit table:
the 4-column pass of the sliced layout, whose ring and consumer groups depend on the number of
outputs.  Empty stencils, poles wider than a stage, scattered tables, partial last slices; tolerance:
the rounding bound of two summation orders (test_gpu_sliced_layout)."""
import numpy as np
import pytest

from gpu_util import torch_cuda
from test_gpu_sliced_layout import _check, _table


@pytest.mark.gpu
@pytest.mark.parametrize("nout", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("length,stride,n,poles", [(3, 4, 5003, 0), (4, 4, 70001, 0),
                                                   (3, 4, 9001, 97), (1, 4, 33, 0),
                                                   (3, 3, 120001, 0)])
def test_narrow_rows_every_output_count(nout, length, stride, n, poles):
    torch = torch_cuda()
    rng = np.random.default_rng(1000 * nout + n)
    # the last case is large enough (2^20 entries) for its unaligned rows to be padded
    sizes, offsets, idx, ws = _table(rng, n, 3000, 20, empty_every=41, pole_every=poles,
                                     scatter=True)
    _check(torch, n, 3000, length, sizes, offsets, idx, ws, nout=nout, seed=nout,
           src_desc=(0, length, stride), dst_descs=[(0, length, length)] * nout)
