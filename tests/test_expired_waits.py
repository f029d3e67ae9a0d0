"""The kernels whose shared memory is filled by bulk copies leave, at an expired wait too, only when
their copies have been waited for (each with a limit again): the memory is another CTA's afterwards.

Checked on the sources, since a copy that never comes cannot be made: every way out of a producer, and
of a warp that feeds itself, runs a drain; the drains' stages and parities, which are computed as
the fills', are walked over all states of a ring.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "opensubdiv_gb300", "csrc")


def _code(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def _block(text, at):
    """The braces' content from the first brace at or behind `at`."""
    start = text.index("{", at)
    depth, end = 0, start
    while True:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        if depth == 0:
            return text[start:end + 1]
        end += 1


def _returns_drained(block):
    outs = list(re.finditer(r"\breturn\s*;", block))
    assert outs
    for m in outs:
        before = block[:m.start()].rstrip()
        assert re.search(r"drain(<S>)?\([^;]*\);$", before), block[max(0, m.start() - 200):m.end()]


@pytest.mark.parametrize("name,kernels", [("stencils_tma.cu", 2), ("stencils_batch.cu", 1)])
def test_producers(name, kernels):
    text = _code(name)
    blocks = [_block(text, m.end()) for m in re.finditer(r"if \(warp == kConsumers / 32\)", text)]
    assert len(blocks) == kernels
    for b in blocks:
        _returns_drained(b)
        # the stage that tells the consumers of the end counts as filled, another's copy does not
        assert ("0, 0, 1}" in b) == bool(re.search(r"bar_arrive\(&full\[stage\]\);\s*drain\(it \+ 1\);", b))
        assert not re.search(r"drain(<S>)?\((full, )?it \+ 1\)", re.sub(
            r"bar_arrive\(&full\[stage\]\);\s*drain\(it \+ 1\);", "", b))


@pytest.mark.parametrize("name,kernel", [("stencils_units.cu", "k_stencils_units"),
                                         ("stencils_batch.cu", "k_stencils_batch_units")])
def test_warps_that_feed_themselves(name, kernel):
    text = _code(name)
    body = _block(text, text.index(kernel + "(const Args"))
    failing = [m for m in re.finditer(r"if \(!(ring::wait|consume<COLLECT>)\(", body)]
    assert failing
    for m in failing:
        _returns_drained(_block(body, m.end()))
    # nothing is on its way where all queued slices are done with
    assert len(re.findall(r"\breturn\s*;", body)) == len(failing) + 1 + body.count("if (!more) return;")
    assert "if (f.popped == f.pushed) return;" in body


@pytest.mark.parametrize("S", [2, 3, 4])
def test_drain_waits_for_every_copy_on_its_way(S):
    """Tiles k < tiles have been filled in order, those up to `arrived` of the last S in any subset: the
    drain's waits pass exactly for the stages whose copy has arrived."""
    for tiles in range(0, 3 * S + 2):
        last = range(max(tiles - S, 0), tiles)
        for subset in range(1 << len(last)):
            arrived = {k for i, k in enumerate(last) if subset >> i & 1}
            phases = [sum(1 for k in range(s, tiles, S) if k not in last or k in arrived)
                      for s in range(S)]
            passes = {k for k in last if phases[k % S] & 1 != (k // S & 1)}
            assert passes == arrived
