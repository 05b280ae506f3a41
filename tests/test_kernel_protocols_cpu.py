"""Host models of what the warps of a kernel agree on, walked through every order of their steps.

A wait inside these kernels may give up (two seconds of clock, or another warp gave up), so the models let every wait end either way
at any time.  What the kernels do at the places that matter is read from their sources.
"""
import itertools
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "flashdeberta_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def _walk(start, steps):
    """Every state that can be reached; `steps` gives the states after one."""
    seen, todo = {start}, [start]
    while todo:
        state = todo.pop()
        for after in steps(state):
            if after not in seen:
                seen.add(after)
                todo.append(after)
    return seen


# ---- attn_fwd_kernel: work items handed from the TMA warp to the softmax warps --------------------------------------------------
#
# Two softmax warps stand for the eight.  An item is (number of its named barriers, whether it is one at all): none for a padding tile.
# Places of a softmax warp: "wait" (for scores), "sync" (named barrier), "next" (for the next item), "ask" (whether it was handed
# out), "read" (its slot), "done".  Of the TMA warp: "load" (every wait of an item), "free" (the slot's readers), "write", "tell", "done".

ITEMS = ((1, True), (2, True), (0, True), (3, True), (1, True), (0, False))


def _softmax_warps_ask():
    text = _source("attn_fwd_sm100.cu")
    ask = re.search(r"auto next_item_of_all = .*?\n  \};", text, re.S)
    taken = re.findall(r"while \((\w+)\(it\)\);", text.split("= softmax groups =")[1])
    assert len(taken) == 1, "the softmax groups' loop over items is not the one modelled here"
    return bool(ask) and "if (taken + 1u >= n) return false;" in ask.group(0) and taken == ["next_item_of_all"] and \
        "*handed_out = asked + 1u;" in text


def _tma_warp_stops():
    post = re.search(r"wait\(bar\(kBarItemFree \+ slot\), \(\(asked >> 1\) - 1u\) & 1u\);(.*?)sts_v4\(at,", _source("attn_fwd_sm100.cu"), re.S)
    assert post, "the hand-over of items is not the one modelled here"
    return "if (!ok) break;" in post.group(1)


def _takeover_faults(ask, stop):
    """Faults that some order of steps leads to.  ask: a softmax warp that gave up takes the items that were handed out; stop: the TMA
    warp writes no slot whose readers it gave up on."""
    faults = set()
    ready = lambda completed, parity: (completed & 1) != parity  # what a parity wait can tell

    def steps(state):
        (place, asked, ok), warps, slots = state
        after = []
        tma = lambda *t, slots=slots: after.append((t, warps, slots))
        what, told, freed, arrived = slots[asked & 1]
        one = lambda *s: tuple(s if i == asked & 1 else x for i, x in enumerate(slots))
        if place == "load":
            tma("free", asked, ok)
            tma("done", asked, False)
        elif place == "free":
            if asked < 2 or ready(freed, ((asked >> 1) - 1) & 1):
                tma("write", asked, ok)
            if asked >= 2:
                tma("done" if stop else "write", asked, False)
        elif place == "write":
            tma("tell", asked, ok, slots=one(asked + 1, told, freed, arrived))
        elif place == "tell":
            more = ITEMS[asked + 1][1] and ok
            tma("load" if more else "done", asked + 1, ok, slots=one(what, told + 1, freed, arrived))
        for i, (at, item, left, taken, ok) in enumerate(warps):
            def put(*w, slots=slots):
                after.append((state[0], tuple(w if j == i else x for j, x in enumerate(warps)), slots))
            what, told, freed, arrived = slots[taken & 1]
            if at == "wait":
                put("sync" if left else "next", item, left, taken, ok)
                put("sync" if left else "next", item, left, taken, False)
            elif at == "next":
                if ok and ready(told, (taken >> 1) & 1):
                    put("read", item, left, taken, ok)
                put("ask" if ask else "done", item, left, taken, False)
            elif at == "ask" and place == "done":
                put("read" if taken < asked else "done", item, left, taken, ok)
            elif at == "read":
                now = (what, told, freed + 1, 0) if arrived == 1 else (what, told, freed, 1)
                put("wait" if ITEMS[what][1] else "done", what, ITEMS[what][0], taken + 1, ok,
                    slots=tuple(now if j == taken & 1 else x for j, x in enumerate(slots)))
        a, b = warps
        if a[0] == b[0] == "sync":  # the named barrier lets both through
            if a[1] != b[1]:
                faults.add("the warps work on different items")
            after.append((state[0], tuple(("wait" if w[2] > 1 else "next", w[1], w[2] - 1, *w[3:]) for w in warps), slots))
        if not after and (a[0], b[0]) != ("done", "done"):
            faults.add("a warp waits for one that has left")
        return after

    first = ("wait", 0, ITEMS[0][0], 0, True)
    states = _walk((("load", 0, True), (first, first), ((0, 0, 0, 0),) * 2), steps)
    assert any(s[1] == (("done", 5, 0, 5, True),) * 2 for s in states)  # all items, nobody gave up
    return faults


def test_softmax_warps_that_give_up_leave_none_behind():
    """However waits give up, every softmax warp reaches the end: the named barriers of an item have no limit of their own, so the warps
    have to work on the same items."""
    assert _takeover_faults(False, True)  # (the model sees the fault)
    assert _takeover_faults(_softmax_warps_ask(), True) == set()


def test_items_that_are_still_to_be_read_are_not_written_over():
    """A TMA warp that gives up on the readers of a slot leaves what is in it: a warp that comes late reads the item that the others read."""
    assert _takeover_faults(True, False)  # (the model sees the fault)
    assert _takeover_faults(True, _tma_warp_stops()) == set()


# ---- encoder_small_kernel: the score buffers of attention_row ----------------------------------------------------------------------
#
# Four warps share a (row, head); two stand for them.  A row of a sequence: each writes scores, all meet, each reads the scores of all.
# A row of no sequence does none of it.


def _buffers_change_with_the_barrier():
    text = _source("encoder_small.cu")
    loop = re.search(r"for \(int item = [^{]*\{.*?attention_row\(.*?\n    \}", text, re.S)
    assert loop and "scores + turn * 64" in loop.group(0), "the loop over rows and heads is not the one modelled here"
    return "turn ^= 1) {" not in loop.group(0) and "if (len > 0) turn ^= 1;" in loop.group(0)


def _scores_written_over(rows, with_barrier):
    """Whether some order of steps lets a warp write a score buffer that the other one still has to read."""
    turns, turn = [], 0
    for full in rows:
        turns.append(turn)
        turn ^= full or not with_barrier
    program = [(step, i) for i, full in enumerate(rows) if full for step in ("write", "meet", "read")]
    found = []

    def steps(state):
        after = []
        for w in (0, 1):
            me, other = state[w], state[1 - w]
            if me == len(program):
                continue
            step, row = program[me]
            if step == "meet" and other < me:
                continue
            if step == "write" and any(what == "read" and turns[row] == turns[r] and r < row for what, r in program[other:]):
                found.append(rows)
            after.append((me + 1, other) if w == 0 else (other, me + 1))
        return after

    _walk((0, 0), steps)
    return bool(found)


def test_scores_of_a_row_are_read_before_they_are_written_over():
    """Whichever rows belong to no sequence (fewer SMs than this kernel usually runs on leave a group of warps more than two of them)."""
    rows = list(itertools.product((False, True), repeat=5))
    assert any(_scores_written_over(r, False) for r in rows)  # (the model sees the fault)
    assert not any(_scores_written_over(r, _buffers_change_with_the_barrier()) for r in rows)


def test_clock_stamps_are_of_one_item():
    """A CTA works on many items and its roles run ahead of one another: every stamp of a development build says which item it is of."""
    for name, items in (("attn_fwd_sm100.cu", {"taken", "asked"}), ("attn_fwd_far1_sm100.cu", {"0u"})):
        assert set(re.findall(r"FDB_STAMP\((\w+),", _source(name))) == items
    assert "(item) == args.trace_item" in _source("attn_fwd_common.cuh")
