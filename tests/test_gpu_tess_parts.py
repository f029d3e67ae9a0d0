"""How many threads share a tessellation pattern: 8, 4, 2 and 1, the last also in more than one round,
every coord and facet equal to the oracle's bit for bit.

The number follows from the patterns listed (faces of 3 and 4 sides by their rates, every other face
for itself), the rows of blocks and the SMs; it is computed here, and each is shown to occur."""
import numpy as np
import pytest

import oracle
from gpu_util import host, torch_cuda


def _parts(reg, listed, faces, sms):
    """(threads per pattern, rounds) of generate_faces for a launch over `faces` faces."""
    kinds = 4 if reg == 4 else 2
    wide = min(-(-faces // 128), 16 * sms)
    threads = 128 * min(wide, max(8 * sms // (8 * kinds), -(-wide // 8)))
    parts = 8
    while parts > 1 and listed > threads * (8 // parts):
        parts //= 2
    return parts, -(-listed // (threads * (8 // parts)))


@pytest.mark.gpu
@pytest.mark.parametrize("reg,faces,top,facet,want", [
    (4, 3000, 40, 3, 8), (4, 9000, 24, 4, 4), (4, 17000, 24, 3, 2), (4, 60000, 24, 3, 1),
    (4, 330000, 2, 4, 1), (3, 9000, 40, 4, 8), (3, 18000, 40, 3, 4), (3, 36000, 48, 3, 2),
    (3, 90000, 48, 3, 1)])
def test_threads_per_pattern(reg, faces, top, facet, want):
    torch = torch_cuda()
    from opensubdiv_gb300 import bfr
    rng = np.random.default_rng(faces + facet)
    many = faces > 300000  # more patterns than threads: pentagons, whose patterns are never shared
    sizes = np.full(faces, 5 if many else reg, np.int32)
    if reg == 4 and not many:
        sizes[rng.random(faces) < 0.1] = 12
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    rates = rng.integers(1, top + 1, offsets[-1]).astype(np.int32)
    for f in np.nonzero(sizes == 12)[0]:
        rates[offsets[f]: offsets[f + 1]] = rng.integers(1, 4, 12)
    keyed = sizes == reg
    listed = int((~keyed).sum())
    if keyed.any():
        runs = rates[offsets[:-1][keyed][:, None] + np.arange(reg)]
        listed += len(np.unique(runs, axis=0))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    parts, rounds = _parts(reg, listed, faces, sms)
    assert parts == want and (rounds > 1) == many
    o = bfr.TessellationOptions(facet, False)
    m = bfr.MeshTessellation(reg, sizes, rates=rates, rate_offsets=offsets, options=o)
    coords, facets, _ = m.Generate()
    t = oracle.tess_mesh(reg, sizes, offsets, rates, facet, False, threads=8)
    assert np.array_equal(host(m.coord_offsets), t["coord_offsets"])
    assert np.array_equal(host(m.facet_offsets), t["facet_offsets"])
    assert np.array_equal(host(coords).view(np.int32), t["coords"].view(np.int32))
    assert np.array_equal(host(facets), t["facets"])
