"""An entry pass's longest pairs on streamed stripes, with the share above
which a pair goes there pinned from "all" to "the few longest": scores,
overflow blocks (through the tie order and the counters) and CIGARs against
the oracle, one query and batches, at every width."""
import numpy as np
import pytest

from libssa_b200 import workloads as W
from test_wide_entry import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [0, 40, 400])
@pytest.mark.parametrize("width", [8, 16, 64])
def test_longest_pairs(built_library, monkeypatch, width, share):
    monkeypatch.setenv("SSA_B200_STREAM_SHARE", str(share))
    rng = np.random.default_rng(31 + share)
    queries = [W.random_residues(rng, n, W.AA20) for n in (30, 128, 129, 260, 700)]
    records = [W.random_residues(rng, int(n), W.AA20) for n in rng.integers(1, 700, 60)]
    # overflows at the start, in the middle and at the end of long records, in
    # one sequence of a register pair or both, and lengths around the blocks
    for q in queries[1:]:
        for n, at in ((900, 0), (901, 400), (902, 700), (903, 901 - len(q)), (2050, 1500), (2051, None)):
            r = W.random_residues(rng, max(n, len(q)), W.AA20)
            if at is not None:
                at = max(0, min(at, len(r) - len(q)))
                r[at:at + len(q)] = W.mutate(rng, q, W.AA20, 0.05, 0.0, (1, 1))
            records.append(r)
    records += [np.tile(queries[3], 12), np.zeros(0, np.uint8)]
    _check(dict(algo="sw", width=width, align=1, hits=16, gap=(-11, -1), chunk=25, simd=2,
                records=[r.tobytes() for r in records], queries=[q.tobytes() for q in queries]))


@pytest.mark.parametrize("share", [None, 0, 40])
@pytest.mark.parametrize("width", [8, 16, 64])
def test_needleman_wunsch_pairs(built_library, monkeypatch, width, share):
    """Needleman-Wunsch on the streamed stripes: a query without a partner
    whole, batches from "all" to "the longest"; records around the blocks, one
    register half ending long before the other, and records past the exact
    16-bit range, which go to the lane emulation."""
    if share is not None:
        monkeypatch.setenv("SSA_B200_STREAM_SHARE", str(share))
    rng = np.random.default_rng(41 + width)
    queries = [W.random_residues(rng, n, W.AA20) for n in (1, 30, 127, 128, 129, 300)]
    records = [W.random_residues(rng, int(n), W.AA20) for n in rng.integers(1, 600, 50)]
    records += [W.random_residues(rng, n, W.AA20) for n in (1, 2, 3, 4, 5, 61, 62, 63, 64, 65, 66, 1500, 2600, 9000)]
    records += [W.mutate(rng, q, W.AA20, 0.1, 0.03, (1, 5)) for q in queries for _ in range(3)]
    _check(dict(algo="nw", width=width, align=1, hits=14, gap=(-11, -1), chunk=25, simd=2,
                records=[r.tobytes() for r in records], queries=[q.tobytes() for q in queries]))


@pytest.mark.parametrize("rows", [5, 6])
@pytest.mark.parametrize("width", [8, 64])
def test_rows_per_lane(built_library, monkeypatch, width, rows):
    """Stripes of 160 and 192 rows: queries around one and two of them, every
    pair of the entry and the re-queued ones there."""
    monkeypatch.setenv("SSA_B200_STREAM_SHARE", "0")
    monkeypatch.setenv("SSA_B200_STREAM_ROWS", str(rows))
    rng = np.random.default_rng(51 + rows)
    s = 32 * rows
    queries = [W.random_residues(rng, n, W.AA20) for n in (1, rows - 1, rows, rows + 1, s - 1, s, s + 1, 2 * s, 2 * s + 1)]
    records = [W.random_residues(rng, int(n), W.AA20) for n in rng.integers(1, 400, 40)]
    records += [W.random_residues(rng, n, W.AA20) for n in (61, 62, 63, 64, 65, 66, 127, 1500)]
    for q in queries[4:]:
        for n in (len(q), 1000, 1003):
            records.append(W.mutate(rng, np.tile(q, n // len(q) + 1)[:n], W.AA20, 0.03, 0.01, (1, 4)))
    _check(dict(algo="sw", width=width, align=1, hits=16, gap=(-11, -1), chunk=25, simd=2,
                records=[r.tobytes() for r in records], queries=[q.tobytes() for q in queries]))
