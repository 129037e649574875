"""How the consumer warps of a decode launch leave the walk through the phases when a record comes late.

The warps of a CTA meet at a barrier without a limit in every phase, and a record that does not come within the
limit ends the walk.  All schedules of a small model of ``consume_launch`` (``csrc/mb_decode.cu``): the record of any
phase arrives at any moment or never, and whoever waits for one may find the limit exceeded at any moment before.
No schedule may leave a warp at the barrier for good.
"""

import pytest

WARPS, PHASES = 3, 3


def _steps_each_warp_decides(state):
    """Every warp waits for the record of its phase by itself and leaves if its own limit runs out."""
    records, warps, _ = state
    for w, (phase, at) in enumerate(warps):
        if at != "top" or phase == PHASES:
            continue
        move = lambda to: (records, warps[:w] + (to,) + warps[w + 1:], ())
        if phase in records:
            yield move((phase, "barrier"))
        else:
            yield move((PHASES, "left"))


def _steps_one_thread_decides(state):
    """Warp 0 looks, at the start of phase p, for the record of p + 1 and marks that phase as the end if its limit runs
    out; what it has marked, the others see behind the barrier inside phase p."""
    records, warps, stops = state
    for w, (phase, at) in enumerate(warps):
        if phase == PHASES:
            continue
        move = lambda to, marks=stops: (records, warps[:w] + (to,) + warps[w + 1:], marks)
        if at == "top":
            if phase in stops:
                yield move((PHASES, "left"))
            elif w > 0 or phase + 1 == PHASES:
                assert phase in records   # never looked at before it has come
                yield move((phase, "barrier"))
            else:
                if phase + 1 in records:
                    yield move((phase, "barrier"))
                else:
                    yield move((phase, "barrier"), stops + (phase + 1,))
        elif at == "before":   # ahead of the walk: record 0
            if w > 0:
                yield move((-1, "barrier"))
            else:
                yield move((-1, "barrier"), stops if 0 in records else stops + (0,))


def _stuck(steps, start):
    """States in which somebody is at the barrier and nothing can happen any more."""
    seen, todo, stuck = set(), [start], []
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        records, warps, stops = state
        follow = list(steps(state))
        if all(at == "barrier" for _, at in warps):
            follow.append((records, tuple((phase + 1, "top") for phase, _ in warps), stops))
        todo += follow
        if not follow and any(at == "barrier" for _, at in warps):
            stuck.append(state)
        if len(records) < PHASES:   # records come in order
            todo.append((records + (len(records),), warps, stops))
    assert len(seen) > 20
    return [s for s in stuck if len(s[0]) == PHASES]


def test_a_verdict_per_warp_can_leave_warps_at_the_barrier():
    assert _stuck(_steps_each_warp_decides, ((), ((0, "top"),) * WARPS, ()))


def test_one_verdict_for_all_warps_never_does():
    assert not _stuck(_steps_one_thread_decides, ((), ((-1, "before"),) * WARPS, ()))
