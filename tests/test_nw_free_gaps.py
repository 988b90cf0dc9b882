"""Needleman-Wunsch with a gap of one that costs nothing: the 16-bit lanes'
overflow line wraps to the largest value, so every pair overflows in its first
block, which the tie order and the overflow counters show.  At the 16-bit entry,
and at 16 bits after the 8-bit entry, against the oracle."""
import numpy as np
import pytest

import oracle
from helpers import matrix_table
from libssa_b200 import workloads as W
from test_wide_entry import _check


def test_every_16_bit_lane_overflows():
    rng = np.random.default_rng(3)
    q, d = (rng.integers(1, 20, n).astype(np.uint8) for n in (30, 25))
    for gap, overflows in (((0, 0), True), ((0, -1), False), ((-1, 0), False)):
        cfg = oracle.SearchConfig(algo="nw", bit_width=16, align_type=0, hitcount=1, chunk_size=1, gap_open=gap[0],
                                  gap_extend=gap[1], lanes8=32, lanes16=16, matrix=matrix_table(("builtin", "blosum62")))
        score, overflow, blocks = oracle.lane_result(cfg, 16, q, d)
        assert overflow is overflows and (blocks == 1) is overflows, gap


@pytest.mark.gpu
@pytest.mark.parametrize("gap", [(0, 0), (0, -1), (-1, 0)])
@pytest.mark.parametrize("width", [8, 16, 64])
def test_free_gaps(built_library, width, gap):
    rng = np.random.default_rng(61)
    queries = [W.random_residues(rng, n, W.AA20) for n in (1, 7, 40, 129, 260)]
    # short records of few lengths: many ties, whose order is the order of the reports
    records = [W.random_residues(rng, int(n), W.AA20) for n in rng.integers(1, 12, 150)]
    records += [W.random_residues(rng, int(n), W.AA20) for n in rng.integers(20, 300, 30)]
    _check(dict(algo="nw", width=width, align=1, hits=40, gap=gap, chunk=50, simd=2,
                records=[r.tobytes() for r in records], queries=[q.tobytes() for q in queries]))
