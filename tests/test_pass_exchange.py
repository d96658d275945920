"""The hand-over between the CTAs of a radix pass's cluster (rs_pass_kernel and
rs_scout in bulk_b200/csrc/radix_sort.cu), as a model run through every order in
which its agents can take their steps: each CTA's ranking warps and its scout
must take the groups that the cluster's first CTA hands out, in that order,
whatever waits for whom.  The scout's steps stand in the order of the source."""
from __future__ import annotations

from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parents[1] / "bulk_b200" / "csrc" / "radix_sort.cu"
CTAS = 2
GROUPS = 5  # the last hand-out ends the loop


def _scout_steps() -> tuple[str, ...]:
    text = SOURCE.read_text()
    body = text[text.index("void rs_scout("):]
    body = body[body.index("{"):body.index("\n}\n")]
    at = {"wait": body.index("rs_wait_cluster(&cnt_bar[par]"), "next": body.index("s_next[par]"),
          "send": body.index("rs_push_u32(s_base")}
    return tuple(sorted(at, key=at.get))


# A CTA's ranking warps: counts (and CTA 0's hand-out of the next group) go out, then the positions of the tile
# before are waited for (it is written out), then the cluster's counts and the next group.
MAIN = ("send", "before", "counts")


def _explore(scout_steps):
    """Every reachable state; returns the first group an agent takes out of order, or None."""
    # state: per CTA (iteration, step) of the main warps and of the scout, the scout's unread next group,
    # s_next by parity, and completed phases and arrivals of the count and position barriers by parity
    def start():
        cta = ((0, 0), (0, 0), (-1, -1), (0, 0), (0, 0), (0, 0), (0, 0))
        return (cta,) * CTAS

    def arrive(done, here, par, need):
        here = list(here)
        done = list(done)
        here[par] += 1
        if here[par] == need:
            here[par] = 0
            done[par] += 1
        return tuple(done), tuple(here)

    def passed(done, par, phase):  # a parity wait: the phase of that parity is over
        return (done[par] & 1) != phase

    seen, todo = set(), [start()]
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        for c in range(CTAS):
            main, scout, nxt, cdone, chere, bdone, bhere = state[c]
            # ---- the ranking warps
            it, step = main
            par, phase = it & 1, (it >> 1) & 1
            if it <= GROUPS:
                new = [list(x) for x in state]
                ok = True
                if MAIN[step] == "send":
                    if it < GROUPS:
                        for q in range(CTAS):
                            new[q][3], new[q][4] = arrive(new[q][3], new[q][4], par, CTAS)
                            if c == 0:
                                n = list(new[q][2])
                                n[par] = it + 1
                                new[q][2] = tuple(n)
                elif MAIN[step] == "before":
                    ok = it == 0 or passed(bdone, par ^ 1, ((it - 1) >> 1) & 1)
                else:
                    ok = it == GROUPS or passed(cdone, par, phase)
                    if ok and it < GROUPS and nxt[par] != it + 1:
                        return ("ranking warps", c, it, nxt[par])
                if ok:
                    new[c][0] = (it, step + 1) if step + 1 < len(MAIN) else (it + 1, 0)
                    todo.append(tuple(tuple(x) for x in new))
            # ---- the scout
            it, step = scout
            par, phase = it & 1, (it >> 1) & 1
            if it < GROUPS:
                new = [list(x) for x in state]
                ok = True
                if scout_steps[step] == "wait":
                    ok = passed(cdone, par, phase)
                elif scout_steps[step] == "next":
                    if nxt[par] != it + 1:
                        return ("scout", c, it, nxt[par])
                else:
                    for q in range(CTAS):
                        new[q][5], new[q][6] = arrive(new[q][5], new[q][6], par, CTAS)
                if ok:
                    new[c][1] = (it, step + 1) if step + 1 < len(scout_steps) else (it + 1, 0)
                    todo.append(tuple(tuple(x) for x in new))
    ends = [s for s in seen if all(x[0][0] > GROUPS and x[1][0] == GROUPS for x in s)]
    assert ends, "no order of steps ends"
    return None


def test_every_agent_takes_the_groups_in_order():
    assert _explore(_scout_steps()) is None


@pytest.mark.parametrize("steps", [("wait", "send", "next"), ("next", "wait", "send")])
def test_the_model_tells_wrong_orders(steps):
    assert _explore(steps) is not None
