"""The handshake between the scan's state warps and the warp that stores their panels, over every interleaving of the two.

A barrier is waited for by the parity of one of its phases: a waiter that is two phases late sees the parity it started with and
waits for good.  The barrier an arrival or a wait names, and the parity it waits for, are taken from the kernel's source."""

import os
import re

from conftest import ROOT

SOURCE = os.path.join(ROOT, "experiment_swa_kda_b200", "csrc", "kda_tc_pscan.cu")


def _handshake():
    src = open(SOURCE).read()
    src = src[src.index("tc_affine_scan_kernel(const"):src.index("split scans, second pass")]

    def one(pattern):
        found = re.findall(pattern, src)
        assert len(found) == 1, (pattern, found)
        return found[0]

    index = r"bar_%s(?:\[([^\]]*)\])?"
    wait = r"mbar_wait\(&" + index + r", (.*?), p\.status"
    expr = lambda text: eval("lambda c: " + (text or "0"))
    return {"pan": (expr(one(r"warp_arrive\(&" + index % "pan" + r", lane\)")), *map(expr, one(wait % "pan"))),
            "out": (expr(one(r"mbar_arrive\(&" + index % "out" + r"\)")), *map(expr, one(wait % "out")))}


def _stuck(handshake, panels):
    """A reachable state in which neither side can go on and not both have ended, or None."""
    pan_give, pan_at, pan_parity = handshake["pan"]
    out_give, out_at, out_parity = handshake["out"]
    state, store = [], []
    for c in range(panels):
        if c > 1:
            state.append(("wait", "out", out_at(c), out_parity(c)))
        state.append(("give", "pan", pan_give(c)))
        store += [("wait", "pan", pan_at(c), pan_parity(c)), ("give", "out", out_give(c))]
    seen, todo = set(), [(0, 0, (0,) * 4)]
    slot = lambda name, i: ("pan", "out").index(name) * 2 + i
    while todo:
        at = todo.pop()
        if at in seen:
            continue
        seen.add(at)
        moved = False
        for side, program in enumerate((state, store)):
            if at[side] == len(program):
                continue
            kind, name, i, *parity = program[at[side]]
            count = list(at[2])
            if kind == "give":
                count[slot(name, i)] += 1
            elif count[slot(name, i)] % 2 == parity[0]:      # the phase of this parity is still open
                continue
            moved = True
            todo.append((at[0] + (side == 0), at[1] + (side == 1), tuple(count)))
        if not moved and at[:2] != (len(state), len(store)):
            return at
    return None


def test_no_interleaving_leaves_a_panel_waiting():
    handshake = _handshake()
    for panels in (1, 2, 3, 4, 9):
        assert _stuck(handshake, panels) is None


def test_one_barrier_for_both_buffers_would_lose_a_panel():
    handshake = _handshake()
    handshake["pan"] = (lambda c: 0, lambda c: 0, lambda c: c & 1)
    assert _stuck(handshake, 1) is None and _stuck(handshake, 4) is not None
