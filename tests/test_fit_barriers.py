"""The barriers of the exercise fit's CTA (csrc/american.cu, lsm_fit_kernel), modelled: a factorer, a
solver and two walkers go through their dates, their waits for the other CTAs end well or badly at
any time, and every interleaving is followed. A named barrier counts its arrivals, so one that a warp
no longer comes to holds the others for good: with the kernel's order of words and barriers no
interleaving is left waiting, and no barrier gets an arrival too many. Warps that return where their
wait fails, each for itself, do get stuck in this model, so it sees such a fault.
"""
import pytest

SIZES = {"X": 3, "Y": 3, "P": 3, "F": 2, "end": 4}  # arrivals that complete a barrier (a warp counts one)


def program(role, dates, all_leave_together):
    """A role's operations, with ("if", flag, value, label) jumping to a label when flag == value."""
    ops, labels = [], {}
    op = ops.append

    def label(name):
        labels[name] = len(ops)

    def gives_up(word, t):  # a wait for the other CTAs, which may fail
        op(("wait",))
        op(("if", "ok", 1, "waited%d" % t))
        op(("set", word))
        label("waited%d" % t)

    if role in ("walker 1", "walker 2"):
        op(("arrive", ("X", dates % 2)))
    for t in range(dates, 0, -1):
        x, f = ("X", t % 2), ("F", t % 2)
        if role == "factorer":
            op(("sync", x))
            if all_leave_together:
                op(("and not", "stop"))
                op(("if", "ok", 0, "idle%d" % t))
                gives_up("lost", t)
                label("idle%d" % t)
                op(("arrive", f))
            else:
                gives_up("stop", t)
                op(("arrive", f))
                op(("if", "ok", 0, "out"))
        elif role == "solver":
            op(("sync", "Y"))
            if all_leave_together:
                op(("if", "ok", 0, "idle%d" % t))
                op(("wait",))
                label("idle%d" % t)
                op(("sync", f))
                op(("and not", "lost"))
                op(("if", "ok", 1, "goes on%d" % t))
                op(("set", "stop"))
                label("goes on%d" % t)
                op(("arrive", "P"))
            else:
                gives_up("stop", t)
                op(("sync", f))
                op(("and not", "stop"))
                op(("arrive", "P"))
                op(("if", "ok", 0, "out"))
        else:
            if t < dates:
                op(("sync", "P"))
                op(("and not", "stop"))
                if not all_leave_together:
                    op(("if", "ok", 0, "out"))
            op(("arrive", "Y"))
            if t > 1:
                op(("arrive", ("X", (t - 1) % 2)))
    if role.startswith("walker"):
        op(("sync", "P"))
    if all_leave_together:
        op(("sync", "end"))
    label("out")
    op(("done",))
    return ops, labels


def stuck_interleavings(dates, all_leave_together):
    roles = ("factorer", "solver", "walker 1", "walker 2")
    progs = [program(r, dates, all_leave_together) for r in roles]
    # places, each role's ok, words set, arrivals at barriers, barrier each role waits at
    start = ((0,) * 4, (1,) * 4, frozenset(), frozenset(), (None,) * 4)
    seen, todo, stuck = {start}, [start], 0
    while todo:
        at, oks, words, arrived, waiting = todo.pop()
        nxt = []
        for k, (ops, labels) in enumerate(progs):
            o = ops[at[k]]
            if waiting[k] is not None or o[0] == "done":
                continue
            count, w, wt = dict(arrived), words, list(waiting)
            place, ok = at[k] + 1, (oks[k],)
            if o[0] in ("sync", "arrive"):
                b = o[1]
                size = SIZES[b[0] if isinstance(b, tuple) else b]
                count[b] = count.get(b, 0) + 1
                assert count[b] <= size
                if o[0] == "sync":
                    wt[k] = b
                if count[b] == size:
                    del count[b]
                    wt = [None if x == b else x for x in wt]
            elif o[0] == "wait":
                ok = (1, 0)
            elif o[0] == "set":
                w = words | {o[1]}
            elif o[0] == "and not":
                ok = (int(oks[k] and o[1] not in words),)
            elif o[0] == "if" and oks[k] == o[2]:
                place = labels[o[3]]
            for v in ok:
                nxt.append((at[:k] + (place,) + at[k + 1:], oks[:k] + (v,) + oks[k + 1:], w,
                            frozenset(count.items()), tuple(wt)))
        stuck += not nxt and any(x is not None for x in waiting)
        for n in nxt:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return stuck


@pytest.mark.parametrize("dates", [1, 2, 3, 4, 5, 8])
def test_no_interleaving_of_failed_waits_is_left_waiting(dates):
    assert stuck_interleavings(dates, True) == 0


def test_warps_that_return_for_themselves_are_left_waiting():
    assert stuck_interleavings(3, False) > 0
