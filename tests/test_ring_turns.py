"""The rings of the staged EvalStencils kernels: one producer fills S stages with tiles in order,
G consumer groups take turns on the tiles, copies of different stages complete in any order, and a
group waits for its tile by the parity of its stage's use.

All interleavings of a model of that protocol are walked.  By parity alone a group can pass before
its tile is there exactly where S is not a multiple of G; with the tiles numbered (Turns in
stencils_tma.cu) it cannot, and every walk comes to its end.  The kernels wait through Turns.
"""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                      "opensubdiv_gb300", "csrc", "stencils_tma.cu")
TILES = 11


def _walk(S, G, numbered):
    """(a group passed a wait early, a state without a next step before the end)."""
    # producer's next tile; per stage: phases completed, a copy on its way, tiles consumed, number;
    # per group: its next tile, whether it has seen the number
    start = (0, ((0, False, 0, -1),) * S, tuple((g, False) for g in range(G)))
    seen, todo, early, stuck = {start}, [start], False, False
    while todo:
        p, stages, groups = todo.pop()
        nxt = []
        if p < TILES and stages[p % S][2] == p // S and not stages[p % S][1]:
            done, _, used, _ = stages[p % S]
            st = list(stages)
            st[p % S] = (done, True, used, p)
            nxt.append((p + 1, tuple(st), groups))
        for s, (done, flying, used, number) in enumerate(stages):
            if flying:
                st = list(stages)
                st[s] = (done + 1, False, used, number)
                nxt.append((p, tuple(st), groups))
        for g, (it, told) in enumerate(groups):
            if it >= TILES:
                continue
            done, flying, used, number = stages[it % S]
            gr = list(groups)
            if numbered and not told:
                if number == it:
                    gr[g] = (it, True)
                    nxt.append((p, stages, tuple(gr)))
                continue
            if (done & 1) == (it // S & 1):  # the phase of this parity is the one in progress
                continue
            if done != it // S + 1:
                early = True
                continue
            st = list(stages)
            st[it % S] = (done, flying, used + 1, number)
            gr[g] = (it + G, False)
            nxt.append((p, tuple(st), tuple(gr)))
        if not nxt and any(it < TILES for it, _ in groups):
            stuck = True
        for n in nxt:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return early, stuck


@pytest.mark.parametrize("S,G", [(2, 1), (3, 1), (3, 2), (3, 3), (4, 2), (4, 3), (4, 4)])
def test_groups_pass_only_when_their_tile_is_there(S, G):
    assert _walk(S, G, False)[0] == (S % G != 0)
    assert _walk(S, G, S % G != 0) == (False, False)
    assert _walk(S, G, True) == (False, False)


def test_kernels_wait_through_turns():
    text = re.sub(r"//[^\n]*", "", open(SOURCE).read())
    turns = text[text.index("struct Turns"):]
    assert "kNumbered = S % G != 0" in turns
    # the barrier of a filled stage is waited for in Turns only, behind the number
    waits = re.findall(r"mbar_wait\(&full\[[^;]*;", text)
    assert len(waits) == 1 and waits[0] in turns[:turns.index("__device__ __forceinline__ void bulk_g2s")]
    kernels = re.split(r"__global__", text)[1:]
    assert len(kernels) == 2
    for k in kernels:
        assert k.count("turns.wait(full, it)") == 1 and k.count("turns.number(") == 1
        # numbered behind the wait for the stage to be empty
        assert k.index("mbar_wait(&empty[") < k.index("turns.number(")
