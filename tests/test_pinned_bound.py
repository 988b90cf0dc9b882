"""Calls whose small arrays or traceback results pass the pinned memory that is
kept for later calls, against the oracle: searches, pairs and repeated calls with
the bound at one byte, at a few kilobytes, and as it is."""
import numpy as np
import pytest

from libssa_b200 import workloads as W
from test_wide_entry import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kept", ["1", "20000", None])
@pytest.mark.parametrize("algo,width", [("sw", 8), ("nw", 16)])
def test_pinned_bound(built_library, monkeypatch, algo, width, kept):
    if kept is not None:
        monkeypatch.setenv("SSA_B200_PINNED_KEPT", kept)
    rng = np.random.default_rng(111)
    queries = [W.random_residues(rng, n, W.AA20) for n in (30, 200, 500)]
    records = [W.mutate(rng, q, W.AA20, 0.1, 0.02, (1, 4)) for q in queries for _ in range(4)]
    records += [W.random_residues(rng, int(n), W.AA20) for n in rng.integers(1, 700, 60)]
    _check(dict(algo=algo, width=width, align=1, hits=20, gap=(-11, -1), chunk=30, simd=2,
                records=[r.tobytes() for r in records], queries=[q.tobytes() for q in queries]))
