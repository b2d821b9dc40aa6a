"""The word through which warp 0 of xg_potrf128 tells the other warps that a
pivot has failed, under every interleaving: per panel warp 0 may write it, all
warps meet at a barrier, each reads it and leaves if it is set; then warp 0
only arrives at a second barrier, on which the others wait, and goes on to the
next panel.  The number of words is read from the source; with one word warp 0
overtakes a warp that has not read it yet, which leaves a panel early, and the
others wait for it without end.  Runs without a GPU (and is the only way to see
this: the margin on the device is a 16-pivot factorisation)."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "exageostat_b200", "csrc",
                   "xg_potrf128.cuh")
PANELS, WARPS = 4, 3


def _words():
    src = open(SRC).read()
    m = re.search(r"__shared__ int s_fail(?:\[(\d+)\])?;", src)
    words = int(m.group(1) or 1)
    if words > 1:  # written and read by the panel's own word
        assert words == 2 and re.search(r"s_fail\[p & 1\] = c0 \+ f;", src)
        assert re.search(r"= s_fail\[p & 1\];", src)
    return words


def _program(warp):
    ops = []
    for p in range(PANELS):
        ops += [("write", p)] if warp == 0 else []
        ops += [("meet", p), ("read", p)]
        ops += [("arrive" if warp == 0 else "wait", p)] if p + 1 < PANELS else []
    return ops + [("done", None)]


def _ends(words, failing):
    """Final states of all interleavings: a tuple per warp, ("left", panel),
    ("done",) or, for a warp that nothing will release, ("stuck", barrier)."""
    prog = [_program(w) for w in range(WARPS)]
    start = ((0,) * WARPS, (0,) * words, (0, 0), (("run",),) * WARPS)
    seen, todo, ends = {start}, [start], set()
    while todo:
        pcs, word, count, state = todo.pop()
        if ("run",) not in state:
            ends.add(state)
            continue
        for w in range(WARPS):
            if state[w] != ("run",):
                continue
            pc, wd, ct, st = list(pcs), list(word), list(count), list(state)
            op, p = prog[w][pc[w]]
            pc[w] += 1
            if op == "done":
                st[w] = ("done",)
            elif op == "write":
                if p == failing:
                    wd[p % words] = 1
            elif op == "read":
                if wd[p % words]:
                    st[w] = ("left", p)
            else:
                bar = 0 if op == "meet" else 1
                ct[bar] += 1
                if op != "arrive":
                    st[w] = ("stuck", bar)
                if ct[bar] == WARPS:
                    ct[bar] = 0
                    st = [("run",) if s == ("stuck", bar) else s for s in st]
            nxt = (tuple(pc), tuple(wd), tuple(ct), tuple(st))
            if nxt not in seen:
                seen.add(nxt)
                todo.append(nxt)
    return ends


@pytest.mark.parametrize("failing", [None] + list(range(PANELS)))
def test_every_warp_leaves_at_the_failing_panel(failing):
    end = ("done",) if failing is None else ("left", failing)
    assert _ends(_words(), failing) == {(end,) * WARPS}


def test_the_model_sees_a_missing_word():
    assert any(("stuck", 1) in e for e in _ends(1, 1))
