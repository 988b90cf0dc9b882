"""stream_columns() and the residue ring of stream_stripes.cuh as they are now,
modelled step by step on the CPU: chunks of STREAM_CHUNK wavefront steps, one
publication per chunk, the progress of the stripe above read in the course of a
chunk and counted from its end, the next chunk's row loaded ahead when it is
there, the column limit a chunk late, the 64-word ring of residues.  Under
random interleavings every block of the row above is read as the stripe above
left it, every lane finds its residue word, every stripe sweeps the columns up
to the final limit, and all tickets finish.  The constants and the order of
the steps are read from the header, so that a change there fails here until the
model follows.  (It takes the place of the older protocol that
test_stream_schedule.py models.)"""
import os
import random
import re

import pytest

HEADER = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "libssa_b200", "csrc",
                           "stream_stripes.cuh")).read()
CHUNK = int(re.search(r"constexpr uint32_t STREAM_CHUNK = (\d+);", HEADER).group(1))
POLL = CHUNK - int(re.search(r"POLL = STREAM_CHUNK - (\d+);", HEADER).group(1))
LAG = int(re.search(r"constexpr uint32_t STREAM_LAG = (\d+);", HEADER).group(1))
DONE = 1 << 31


def test_the_header_has_the_modelled_order():
    body = HEADER[HEADER.index("uint32_t stream_columns("):HEADER.index("// The stripe has ended after")]
    at = 0
    for step in ["last = limit();", "for( uint32_t s0 = 0;; s0 += CHUNK )",
                 "cols = min( cols, (uint32_t) __shfl_sync( 0xffffffffu, last, 0 ) + 1u );", "last = limit();",
                 "if( sp.above && s0 < cols )", "if( !have )", "need = min( s0 + CHUNK, cols )", "if( avail < need )",
                 "stream_wait( sp.above, need", "avail = v & ~STREAM_DONE;", "cols = min( cols, avail );",
                 "pf = __ldcg( sp.row + (uint64_t) s0 * 2", "st.in[lane] = pf;", "s2 = s0 + CHUNK;",
                 "have = s2 < cols && avail >= min( s2 + CHUNK, cols );", "pf = __ldcg( sp.row + (uint64_t) s2 * 2",
                 "steps = cols + 31u;", "if( cols == 0 || s0 >= steps )", "refill( s0 );", "s1 = min( s0 + CHUNK, steps );",
                 "poll = sp.above && avail < cols;", "min( s0 + POLL, s1 )", "seen = load_relaxed( sp.above );",
                 "c < (int32_t) s1 - 31", "__stcg( sp.row", "fence_acq_rel();", "store_relaxed( sp.mine, s1 - 31u );",
                 "avail = max( avail, __shfl_sync( 0xffffffffu, seen, 0 ) & ~STREAM_DONE );", "if( s1 == steps )"]:
        at = body.find(step, at)
        assert at >= 0, step
        at += len(step)
    ring = HEADER[HEADER.index("struct StreamResidues"):HEADER.index("// One stripe's place among")]
    for step in ["ring[lane] = fetch( lane );", "ring[32 + lane] = fetch( lane - 32 );", "next = fetch( 32 + lane );",
                 "if( s0 && lane < (int) STREAM_CHUNK )",
                 "ring[(s0 + 32u - STREAM_CHUNK + (uint32_t) lane) & 63u] = next;", "next = fetch( (int32_t) s0 + 32 + lane );",
                 "ring[b & 63]"]:
        assert step in ring, step


class Ring:
    def __init__(self):
        self.words = [None] * 64
        for lane in range(32):
            self.words[lane] = lane
            self.words[32 + lane] = lane - 32
        self.next = [32 + lane for lane in range(CHUNK)]

    def refill(self, s0):
        if s0:
            for lane in range(CHUNK):
                self.words[(s0 + 32 - CHUNK + lane) & 63] = self.next[lane]
                self.next[lane] = s0 + 32 + lane

    def read(self, b):
        assert self.words[b & 63] == b, (b, self.words[b & 63])


def _sweep(state, ticket, pred, stripe, last_stripe, cols, row, h, cut, ring):
    """One stripe; yields 0 where another warp may run and 1 after a wavefront step."""
    progress, limit = state["progress"], state["limit"]
    above = pred is not None
    avail, have, pf, s0 = 0, False, [], 0
    last = limit[h] if limit is not None else None
    swept = 0
    if ring:
        for lane in range(32):
            ring.read(-lane)                    # the first step's words
    while True:
        if limit is not None:
            cols = min(cols, last + 1)
            last = limit[h]
        if above and s0 < cols:
            if not have:
                need = min(s0 + CHUNK, cols)
                if avail < need:
                    while not (progress[pred] & DONE or progress[pred] >= need):
                        yield 0
                    avail = progress[pred] & ~DONE
                    if avail < need:
                        cols = min(cols, avail)
                yield 0
                pf = [(c, row[c]) for c in range(s0, min(s0 + CHUNK, cols))]
            yield 0
            inbound = list(pf)
            s2 = s0 + CHUNK
            have = s2 < cols and avail >= min(s2 + CHUNK, cols)
            if have:
                pf = [(c, row[c]) for c in range(s2, min(s2 + CHUNK, cols))]
        else:
            inbound = []
        steps = cols + 31
        if cols == 0 or s0 >= steps:
            break
        if ring:
            ring.refill(s0)
        s1 = min(s0 + CHUNK, steps)
        poll, seen = above and avail < cols, 0
        for s in range(s0, s1):
            if s == s0 + POLL and poll:
                seen = progress[pred]
            if above and s < cols:              # lane 0's row above
                assert inbound[s - s0] == (s, stripe - 1), (h, stripe, s, inbound[s - s0])
            if ring:
                for lane in (0, 1, 7, 30, 31):
                    ring.read(s - lane + 1)
            if cut is not None and stripe == cut[0] and s == cut[1] and limit is not None:
                limit[h] = min(limit[h], cut[1])
            yield 1
        swept = max(swept, min(cols, s1))
        if not last_stripe:
            for c in range(max(0, s0 - 31), s1 - 31):
                row[c] = stripe
                if c % 5 == 0:
                    yield 0
            yield 0
            if s1 > 31:
                progress[ticket] = s1 - 31
        if poll:
            avail = max(avail, seen & ~DONE)
        if s1 == steps:
            break
        s0 += CHUNK
    if not last_stripe:
        progress[ticket] = DONE | cols
    return swept, cols


def _tickets(hits):
    """(stripe, hit) in ticket order, and the first ticket of each stripe."""
    order, cum = [], [0]
    for stripe in range(max(n for n, _, _ in hits)):
        order += [(stripe, h) for h, (n, _, _) in enumerate(hits) if n > stripe]
        cum.append(len(order))
    return order, cum


@pytest.mark.parametrize("warps", [1, 2, 5, 13])
@pytest.mark.parametrize("limited", [False, True])
@pytest.mark.parametrize("seed", range(6))
def test_random_interleavings(warps, limited, seed):
    r = random.Random(1000 * warps + 10 * seed + limited)
    hits = sorted([(r.randint(1, 6), r.choice([1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 64, 100, r.randint(1, 200)]), None)
                   for _ in range(r.randint(1, 7))], key=lambda x: -x[0])
    if limited:
        hits = [(n, c, (r.randrange(n), r.randrange(c)) if r.random() < 0.7 else None) for n, c, _ in hits]
    order, cum = _tickets(hits)
    state = {"next": 0, "progress": [0] * len(order), "limit": [1 << 30] * len(hits) if limited else None}
    rows = [[-1] * c for _, c, _ in hits]
    done = {}

    def warp():
        while state["next"] < len(order):
            ticket = state["next"]
            state["next"] += 1
            stripe, h = order[ticket]
            pred = cum[stripe - 1] + h if stripe else None
            n, cols, cut = hits[h]
            done[stripe, h] = yield from _sweep(state, ticket, pred, stripe, stripe == n - 1, cols, rows[h], h, cut, Ring())

    running = [warp() for _ in range(warps)]
    for _ in range(4_000_000):
        if not running:
            break
        w = r.choice(running)
        for _ in range(r.choice([1, 1, 3, 40])):
            try:
                next(w)
            except StopIteration:
                running.remove(w)
                break
    assert not running and len(done) == len(order)
    for (stripe, h), (swept, cols) in done.items():
        n, all_cols, cut = hits[h]
        # a stripe may end at the limit that it knows of, or have gone past it; never before the final one
        final = all_cols if cut is None or not limited else cut[1] + 1
        assert min(final, all_cols) <= cols <= swept <= all_cols, (stripe, h)


def test_stripes_follow_one_another_at_the_stated_lag():
    """Warps of one speed, one per stripe: stripe i ends i x STREAM_LAG steps after the first."""
    cols, n = 600, 12
    order, cum = _tickets([(n, cols, None)])
    state = {"progress": [0] * n, "limit": None}
    row, ended, t = [-1] * cols, {}, 0
    warps = {i: _sweep(state, i, i - 1 if i else None, i, i == n - 1, cols, row, 0, None, None) for i in range(n)}
    while warps:
        t += 1
        for i in list(warps):
            waited = 0
            try:
                while next(warps[i]) == 0 and waited < 50:     # up to the end of a step, or a wait
                    waited += 1
            except StopIteration:
                ended[i] = t
                del warps[i]
    assert [ended[i + 1] - ended[i] for i in range(n - 1)] == [LAG] * (n - 1)
