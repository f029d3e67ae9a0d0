"""Tessellation patterns of a mesh, each generated by several threads (one per row of runs and
strips) as long as there are few patterns, by one thread when there are many: every coord and facet
equals the oracle's bit for bit on either side of the changes (8, 4, 2 and 1 threads per pattern),
for quad and triangle schemes, faces whose pattern has no key (5 and 12 sides), inner rates, rates
from 1 up and facets of 3 and 4 with and without kept quads.
"""
import numpy as np
import pytest

import oracle
from gpu_util import host, torch_cuda


@pytest.mark.gpu
@pytest.mark.parametrize("reg,faces,top,facet,keep", [
    (4, 1, 7, 3, False), (4, 300, 40, 3, False), (4, 300, 40, 4, True), (4, 4900, 12, 4, False),
    (4, 7000, 9, 4, True), (4, 15000, 9, 3, False), (4, 30000, 7, 4, True),
    (3, 200, 40, 3, False), (3, 13000, 24, 4, False), (3, 45000, 40, 3, False)])
def test_patterns_equal_the_oracles(reg, faces, top, facet, keep):
    torch_cuda()
    from opensubdiv_gb300 import bfr
    rng = np.random.default_rng(faces + facet)
    sizes = np.full(faces, reg, np.int32)
    if reg == 4:
        sizes = rng.choice([4, 4, 4, 4, 4, 3, 5, 12], faces).astype(np.int32)
    inner = np.where(sizes == 4, rng.choice([0, 0, 0, 1, 2], faces), rng.choice([0, 0, 1], faces))
    offsets = np.concatenate([[0], np.cumsum(sizes + inner)]).astype(np.int32)
    rates = rng.integers(1, top + 1, offsets[-1]).astype(np.int32)
    for f in np.nonzero(rng.random(faces) < 0.2)[0]:  # uniform faces
        rates[offsets[f]: offsets[f + 1]] = rates[offsets[f]]
    o = bfr.TessellationOptions(facet, keep)
    m = bfr.MeshTessellation(reg, sizes, rates=rates, rate_offsets=offsets, options=o)
    coords, facets, _ = m.Generate()
    t = oracle.tess_mesh(reg, sizes, offsets, rates, facet, keep, threads=8)
    assert np.array_equal(host(m.coord_offsets), t["coord_offsets"])
    assert np.array_equal(host(m.facet_offsets), t["facet_offsets"])
    assert np.array_equal(host(coords).view(np.int32), t["coords"].view(np.int32))
    assert np.array_equal(host(facets), t["facets"])
