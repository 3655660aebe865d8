"""The order of the grid-resident reverse steps, played on the host (CPU).

A CTA's reverse step k: wait for the arrivals (the rule under test, taken from
the library), read and later clear an adjoint-ring slot, wait for every CTA's
part of lam_g of step k-1, publish its own part, scatter, arrive.  The slot is
complete, and free to be scattered into two steps later, when every CTA has
done its scatter of step k-2 (k-1 with zero delays).
"""

import ctypes as C
import heapq

import numpy as np
import pytest

from leviathan_v1_b200 import _lib


def _rule(steps, early):
    lib = _lib.load()
    counter, arrivals = C.c_int32(), C.c_int32()
    out = []
    for k in range(steps):
        assert lib.lev_adj_reverse_wait(k, early, C.byref(counter), C.byref(arrivals)) == 0
        out.append((counter.value, arrivals.value))
    return out


def _violations(rule, early, walk, scatter):
    """Steps that a CTA enters (passes its wait) before what it reads is
    complete; walk and scatter: times of shape [CTAs, steps]."""
    G, steps = walk.shape
    count = [0, 0]              # the two arrival counters
    arrived = np.zeros(G, int)  # steps each CTA has arrived for
    parts = np.zeros(steps, int)
    bad = 0
    events = [(walk[c, 0], c, "enter") for c in range(G)]
    heapq.heapify(events)
    waiting = []                # (CTA, stage) that cannot go on yet
    step = np.zeros(G, int)
    now = 0.0
    while events or waiting:
        assert events, "the CTAs wait for each other"
        now, c, stage = heapq.heappop(events)
        waiting.append((c, stage))
        moved = True
        while moved:
            moved = False
            for item in list(waiting):
                c, stage = item
                k = step[c]
                at, want = rule[k]
                if stage == "enter" and count[at] >= want * G:
                    bad += int((arrived < k - (1 if early else 0)).any())
                    waiting[waiting.index(item)] = (c, "parts")
                elif stage == "parts" and (k == 0 or parts[k - 1] == G):
                    parts[k] += 1
                    waiting.remove(item)
                    heapq.heappush(events, (now + scatter[c, k], c, "arrive"))
                elif stage == "arrive":
                    count[at] += 1
                    arrived[c] += 1
                    waiting.remove(item)
                    step[c] += 1
                    if step[c] < steps:
                        heapq.heappush(events, (now + walk[c, step[c]], c, "enter"))
                else:
                    continue
                moved = True
    assert (arrived == steps).all()
    return bad


def _times(seed, G, steps):
    """Walks and scatters of one or two CTAs with long rows among short ones."""
    rng = np.random.default_rng(seed)
    walk = rng.uniform(0.5, 1.5, (G, steps))
    scatter = rng.uniform(0.05, 0.2, (G, steps))
    for c in rng.choice(G, 1 + seed % 2, replace=False):
        scatter[c] *= rng.uniform(5.0, 60.0)
        walk[c] *= rng.uniform(1.0, 6.0)
    return walk, scatter


@pytest.mark.parametrize("early", [1, 0])
def test_no_slot_is_read_before_its_scatters_are_done(early):
    rule = _rule(25, early)
    for seed in range(60):
        walk, scatter = _times(seed, 2 + seed % 9, 25)
        assert _violations(rule, early, walk, scatter) == 0, seed


def test_the_model_sees_one_counter_of_all_steps_fail():
    """One total for all steps, k-1 arrivals per CTA before step k: a fast CTA's
    next arrival stands in for a slow one's missing one."""
    rule = [(0, max(k - 1, 0)) for k in range(25)]
    assert any(_violations(rule, 1, *_times(seed, 2 + seed % 9, 25)) for seed in range(60))
