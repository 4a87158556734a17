"""The LSTM recurrence's gate warps report to its MMA warps through hardware barriers, whose waiting has no limit.  That no
warp is left at one, whoever gives up when, is searched here over every order in which the warps can take their steps: a model
of the exits in lstm_tmem_kernel, with two warps of each kind and any wait that may run out at any time."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gigaslop_b200", "csrc", "lstm.cu")
GATES, MMAS, N = 2, 2, 4                                   # N = threads of the barrier, in warps


def stuck_state(barriers, T):
    """A state in which a warp waits and nothing can happen any more, or None.  `barriers`: the reports of step s go to barrier
    s % barriers.  A warp is (place, step); the rest is the abort flag, commits per step and arrivals per barrier."""
    def arrive(count, waiting, b):
        count = count[:b] + (count[b] + 1,) + count[b + 1:]
        if count[b] == N:                                  # complete: the waiting warps go on, the barrier starts afresh
            return count[:b] + (0,) + count[b + 1:], b
        return count, None

    def release(warps, b):
        return tuple(("m1", s) if place == "at" and (s - 1) % barriers == b else (place, s) for place, s in warps)

    def successors(state):
        gates, mmas, abort, commits, count = state
        for i, (place, s) in enumerate(gates):
            if place == "end":
                continue
            put = lambda w: tuple(sorted(gates[:i] + (w,) + gates[i + 1:]))
            if place == "g0":                              # the ih tile: there, or not in time (or the abort flag is seen)
                yield put(("g1", s)), mmas, abort, commits, count
            elif place == "g1" and commits[s] == MMAS:     # accumulators complete: gate math, report
                nxt = ("g0", s + 1) if s + 1 < T else ("end", 0)
                if s + 1 < T:
                    c, b = arrive(count, mmas, s % barriers)
                    yield put(nxt), (mmas if b is None else tuple(sorted(release(mmas, b)))), abort, commits, c
                else:
                    yield put(nxt), mmas, abort, commits, count
            # gives up: abort flag, and the report all the same
            c, b = arrive(count, mmas, s % barriers) if s + 1 < T else (count, None)
            yield put(("end", 0)), (mmas if b is None else tuple(sorted(release(mmas, b)))), True, commits, c
        for i, (place, s) in enumerate(mmas):
            if place in ("end", "at"):
                continue
            put = lambda w, m=mmas: tuple(sorted(m[:i] + (w,) + m[i + 1:]))

            def gave_up():
                c, b = arrive(count, mmas, s % barriers)
                m = put(("end", 0))
                return gates, (m if b is None else tuple(sorted(release(m, b)))), True, commits, c
            if place == "m0":
                if s == 0:
                    yield gates, put(("m1", 0)), abort, commits, count
                else:                                      # waits for the reports of step s - 1
                    c, b = arrive(count, mmas, (s - 1) % barriers)
                    m = put(("at", s))
                    yield gates, (m if b is None else tuple(sorted(release(m, b)))), abort, commits, c
            elif place == "m1":                            # the other CTAs' h, then the MMAs and their commit
                yield gates, put(("m3", s)), abort, commits[:s] + (commits[s] + 1,) + commits[s + 1:], count
                yield gave_up()
            elif abort:                                    # m3: the flag after the commit
                yield gave_up()
            else:
                yield gates, put(("m0", s + 1) if s + 1 < T else ("end", 0)), abort, commits, count

    start = ((("g0", 0),) * GATES, (("m0", 0),) * MMAS, False, (0,) * T, (0,) * barriers)
    seen, todo = {start}, [start]
    while todo:
        state = todo.pop()
        nxt = list(successors(state))
        if not nxt and any(place != "end" for place, _ in state[0] + state[1]):
            return state
        for n in nxt:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return None


def test_one_barrier_could_leave_a_warp_waiting():
    """The search is sharp: with a single barrier a gate warp's second report can complete the step before."""
    assert stuck_state(1, 4) is not None


@pytest.mark.parametrize("T", [1, 2, 3, 5])
def test_no_warp_is_left_at_the_barriers_of_the_kernel(T):
    src = open(SRC).read()
    body = src[src.index("lstm_tmem_kernel("):src.index("// ---- host")]
    reports, waits = re.findall(r"named_arrive<[^;]*;", body), re.findall(r"named_sync<[^;]*;", body)
    assert len(reports) == 4 and len(waits) == 1           # the exits that the model has
    barriers = 2 if all("(s & 1)" in r or "(gave_up & 1)" in r for r in reports) and "OWN_READY + hb" in waits[0] else 1
    assert stuck_state(barriers, T) is None
