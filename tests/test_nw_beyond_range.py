"""Needleman-Wunsch pairs beyond the exact 16-bit range, which the lane
emulation scores beside the entry pass, or after it when there are many:
records around each query's limit, in batches whose queries have different
limits, with the longest of the others streamed or not; against the oracle, and
where they ran from the timing report."""
import re

import numpy as np
import pytest

from libssa_b200 import workloads as W
from test_scaled_tables import check_scaled
from test_wide_entry import _check

pytestmark = pytest.mark.gpu


def _reported(capfd, monkeypatch, check, *args):
    monkeypatch.setenv("SSA_B200_TIMING", "1")
    capfd.readouterr()
    check(*args)
    return re.findall(r"(\d+) pairs beyond the 16-bit range, (\w+) the entry pass", capfd.readouterr().err)


@pytest.mark.parametrize("share", [None, 0, 40])
@pytest.mark.parametrize("width", [16, 64])
def test_records_around_the_limit(built_library, monkeypatch, capfd, width, share):
    """Limits (a step of 11 at most, 30,000 less two openings in all): 2,725
    columns less the query's rows, rounded up to whole passes or stripes."""
    if share is not None:
        monkeypatch.setenv("SSA_B200_STREAM_SHARE", str(share))
    rng = np.random.default_rng(71)
    queries = [W.random_residues(rng, n, W.AA20) for n in (20, 300, 700, 900, 1100)]
    limits = sorted({2725 - 4 - m for n in (300, 700, 900, 1100) for r in (64, 80, 96, 112, 128)
                     for m in (-(-n // r) * r,)})
    records = [W.random_residues(rng, n + d, W.AA20) for n in limits for d in (-1, 0, 1)]
    records += [W.random_residues(rng, int(n), W.AA20) for n in rng.integers(1, 600, 40)]
    records += [W.random_residues(rng, n, W.AA20) for n in (2700, 2721, 4000)]
    found = _reported(capfd, monkeypatch, _check,
                      dict(algo="nw", width=width, align=0, hits=25, gap=(-11, -1), chunk=30, simd=2,
                           records=[r.tobytes() for r in records], queries=[q.tobytes() for q in queries]))
    assert max(int(n) for n, _ in found) > 20 and all(where == "beside" for _, where in found)


@pytest.mark.parametrize("cap", [None, "700"])
def test_many(built_library, monkeypatch, capfd, cap):
    """16 x BLOSUM62, a step of 176 at most: a limit of 170 columns less the
    query's rows, which 10,500 pairs exceed; in one list, and in lists of 700."""
    if cap is not None:
        monkeypatch.setenv("SSA_B200_REQUEUE_CAP", cap)
    rng = np.random.default_rng(72)
    queries = [W.random_residues(rng, n, W.AA20) for n in (41, 45, 50, 55, 60)]
    records = [W.random_residues(rng, int(n), W.AA20) for n in rng.integers(140, 160, 2100)]
    records += [W.random_residues(rng, int(n), W.AA20) for n in rng.integers(1, 90, 40)]
    found = _reported(capfd, monkeypatch, check_scaled,
                      dict(algo="nw", width=16, align=0, hits=20, gap=(-11, -1), chunk=1000, simd=1, records=records,
                           queries=queries), 16)
    assert ("10500", "after") in found and ("2100", "beside") in found
