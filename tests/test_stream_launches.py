"""Streamed pairs whose boundary rows and ticket words do not fit one launch:
a memory limit of a few items, at every width, for the longest pairs of an entry
pass and the re-queued ones, against the oracle."""
import re

import numpy as np
import pytest

from libssa_b200 import workloads as W
from test_wide_entry import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("memory", [1, 9000, 60000])
@pytest.mark.parametrize("algo,width", [("sw", 8), ("sw", 16), ("sw", 64), ("nw", 8), ("nw", 16), ("nw", 64)])
def test_several_launches(built_library, monkeypatch, capfd, algo, width, memory):
    """1: a launch per item; 9,000: a few items of the longest query and more of
    the shorter ones (a record of 300 against 260 rows takes 2,400 bytes)."""
    monkeypatch.setenv("SSA_B200_STREAM_SHARE", "0")
    monkeypatch.setenv("SSA_B200_STREAM_MEMORY", str(memory))
    monkeypatch.setenv("SSA_B200_TIMING", "1")
    rng = np.random.default_rng(101)
    queries = [W.random_residues(rng, n, W.AA20) for n in (40, 128, 129, 260, 500)]
    records = [W.random_residues(rng, int(n), W.AA20) for n in rng.integers(1, 500, 30)]
    records += [W.random_residues(rng, n, W.AA20) for n in (1200, 900)]
    for q in queries:
        for n in (len(q), 600, 603):
            records.append(W.mutate(rng, np.tile(q, n // len(q) + 1)[:n], W.AA20, 0.03, 0.01, (1, 4)))
    capfd.readouterr()
    _check(dict(algo=algo, width=width, align=1, hits=14, gap=(-11, -1), chunk=25, simd=2,
                records=[r.tobytes() for r in records], queries=[q.tobytes() for q in queries]))
    found = re.findall(r"(\d+) items on streamed stripes in (\d+) launches", capfd.readouterr().err)
    assert found and max(int(launches) for _, launches in found) > (1 if memory > 9000 else 3)
    assert memory > 1 or all(items == launches for items, launches in found)
