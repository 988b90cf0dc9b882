"""The schedule of stream_stripes.cuh, modelled step by step on the CPU: warps
take (stripe, alignment) tickets stripe by stripe, follow the stripe above
through the boundary row that is updated in place, prefetch 32 columns of it
when they are there, publish their progress every 32 columns and may end early
at a column limit.  Under random interleavings, with any number of warps, every
boundary column is read as the stripe above left it, every stripe sweeps the
columns up to the final limit, and all tickets finish."""
import random

import pytest

DONE = 1 << 31


def _ticket_stripe(cum, ticket):
    lo, hi = 0, len(cum) - 1
    while hi - lo > 1:
        mid = (lo + hi) // 2
        if cum[mid] <= ticket:
            lo = mid
        else:
            hi = mid
    return lo


def _warp(state, cum, hits):
    """One warp as a generator: yields wherever another warp may run."""
    n_tickets = cum[-1]
    while True:
        ticket = state["next"]
        state["next"] += 1
        if ticket >= n_tickets:
            return
        stripe = _ticket_stripe(cum, ticket)
        h = ticket - cum[stripe]
        pred = cum[stripe - 1] + h if stripe else None
        n_stripes, cols, cut = hits[h]
        row, progress, limit = state["row"][h], state["progress"], state["limit"]
        last = stripe == n_stripes - 1
        avail, have, pf, s0, swept = 0, False, [], 0, 0
        while True:
            if limit is not None:
                cols = min(cols, limit[h] + 1)
            if pred is not None and s0 < cols:
                if not have:
                    need = min(s0 + 32, cols)
                    if avail < need:
                        while not (progress[pred] & DONE or progress[pred] >= need):
                            yield
                        avail = progress[pred] & ~DONE
                        if avail < need:
                            cols = min(cols, avail)
                    pf = [(c, row[c]) for c in range(s0, min(s0 + 32, cols))]
                for c, writer in pf:
                    assert writer == stripe - 1, (h, stripe, c, writer)
                have = False
                yield
                if s0 + 32 < cols:
                    need = min(s0 + 64, cols)
                    avail = max(avail, progress[pred] & ~DONE)
                    if avail >= need:
                        pf = [(c, row[c]) for c in range(s0 + 32, min(s0 + 64, cols))]
                        have = True
            steps = cols + 31
            if cols == 0 or s0 >= steps:
                break
            s1 = min(s0 + 32, steps)
            swept = max(swept, min(cols, s1))
            if limit is not None and cut is not None and stripe == cut[0] and s0 <= cut[1] < s1:
                limit[h] = min(limit[h], cut[1])       # a candidate in that column
            yield
            if not last:
                for c in range(max(0, s0 - 31), s1 - 31):
                    row[c] = stripe
                yield
                if s1 > 31:
                    progress[ticket] = s1 - 31
            if s1 == steps:
                break
            s0 += 32
        yield
        if pred is not None:
            while not progress[pred] & DONE:
                yield
        state["swept"][(h, stripe)] = swept
        if not last:
            progress[ticket] = DONE | cols


@pytest.mark.parametrize("limited", [False, True])
@pytest.mark.parametrize("warps", [1, 3, 40])
@pytest.mark.parametrize("seed", range(6))
def test_stream_schedule(seed, warps, limited):
    rng = random.Random(100 * seed + warps + limited)
    hits = sorted(([rng.randint(1, 9), rng.choice([1, 2, 31, 32, 33, 63, 64, 65, 97, rng.randint(1, 400)]), None]
                   for _ in range(rng.randint(1, 6))), key=lambda t: -t[0])
    for t in hits:
        if rng.random() < 0.7:
            t[2] = (rng.randrange(t[0]), rng.randrange(t[1]))
    cum = [0]
    for i in range(hits[0][0]):
        cum.append(cum[-1] + sum(t[0] > i for t in hits))
    state = {"next": 0, "row": [[None] * t[1] for t in hits], "progress": [0] * cum[-1],
             "limit": [0x7f7f7f7f] * len(hits) if limited else None, "swept": {}}
    running = [_warp(state, cum, hits) for _ in range(warps)]
    for _ in range(2_000_000):
        if not running:
            break
        k = rng.randrange(len(running))
        try:
            next(running[k])
        except StopIteration:
            running.pop(k)
    assert not running, "the schedule did not finish"
    assert len(state["swept"]) == cum[-1]
    for h, (n, cols, _) in enumerate(hits):
        final = min(cols, state["limit"][h] + 1) if limited else cols
        assert all(state["swept"][(h, i)] >= final for i in range(n)), h
