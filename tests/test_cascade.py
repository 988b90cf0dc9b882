"""The 8-bit entry's re-queued pairs in the 16-bit pass: Smith-Waterman on
streamed stripes of two sequences per register (odd counts, lengths around the
4-column blocks and the 16-block chunks, queries around the stripes of 128 and
256 rows, scores past the 16x2 range and past 65,535), Needleman-Wunsch over
all pairs when most overflow and over the list when few do, against the oracle
with the overflow counters."""
import numpy as np
import pytest

from libssa_b200 import workloads as W
from test_wide_entry import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 2, 7])
def test_sw_requeued_pairs(built_library, copies):
    rng = np.random.default_rng(20 + copies)
    queries = [W.random_residues(rng, n, W.AA20) for n in (60, 127, 128, 129, 256, 257, 700)]
    records = []
    for q in queries:
        for k in range(copies):
            n = [len(q), 1000, 63, 64, 65, 2047, 2052][k]
            records.append(W.mutate(rng, np.tile(q, n // len(q) + 1)[:max(n, 60)], W.AA20, 0.02, 0.0, (1, 1)))
    records += [W.random_residues(rng, int(n), W.AA20) for n in rng.integers(1, 500, 50)]
    _check(dict(algo="sw", width=8, align=1, hits=14, gap=(-11, -1), chunk=20, simd=2,
                records=[r.tobytes() for r in records], queries=[q.tobytes() for q in queries]))


def test_sw_requeued_past_the_16x2_range(built_library):
    records = [b"W" * n for n in (2790, 2791, 2792, 2793, 5957, 5958, 30, 20)]
    _check(dict(algo="sw", width=8, align=0, hits=8, gap=(-11, -1), chunk=3, simd=2, records=records,
                queries=[b"W" * 5959, b"W" * 2792]))


def test_sw_requeued_with_a_table_past_int8(built_library):
    """16 x BLOSUM62 wraps at 8 bits; the 16-bit pass stays with the emulation."""
    rng = np.random.default_rng(22)
    queries = [W.random_residues(rng, n, W.AA20) for n in (50, 300)]
    records = [W.mutate(rng, q, W.AA20, 0.1, 0.02, (1, 3)) for q in queries for _ in range(3)]
    records += [W.random_residues(rng, int(n), W.AA20) for n in rng.integers(1, 300, 30)]
    _check(dict(algo="sw", width=8, align=0, hits=9, gap=(-11, -1), chunk=1000, simd=1,
                records=[r.tobytes() for r in records], queries=[q.tobytes() for q in queries]), 16)


@pytest.mark.parametrize("lens", [(3, 9), (40, 90), (100, 140), (255, 600)])
def test_nw_requeued_pairs(built_library, lens):
    """Query and record lengths from those whose lanes never overflow at 8 bits
    to those that all do in their first block, and records past the exact
    16-bit range."""
    rng = np.random.default_rng(lens[0])
    queries = [W.random_residues(rng, int(n), W.AA20) for n in rng.integers(lens[0], lens[1], 3)]
    records = [W.mutate(rng, q, W.AA20, 0.1, 0.03, (1, 3)) for q in queries for _ in range(4)]
    records += [W.random_residues(rng, int(n), W.AA20) for n in rng.integers(1, 2 * lens[1], 80)]
    records += [W.random_residues(rng, n, W.AA20) for n in (4000, 9000)]
    _check(dict(algo="nw", width=8, align=0, hits=12, gap=(-11, -1), chunk=30, simd=2,
                records=[r.tobytes() for r in records], queries=[q.tobytes() for q in queries]))
