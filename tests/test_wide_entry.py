"""The 16- and 64-bit entries through the 16x2 kernels: Smith-Waterman up to
the score at which a 16-bit half could leave its range (pairs that reach it are
scored by the lane emulation), Needleman-Wunsch at 64 bits within its exact
range, and score tables that do not fit int8 or int16.  Exact, against the
oracle: hits, order, CIGARs, coordinates and overflow counters."""
import os

import numpy as np
import pytest

import oracle
from helpers import DATA, lanes, matrix_table, product_search, product_setup
from libssa_b200 import workloads as W

pytestmark = pytest.mark.gpu

# 16x2 range of the Smith-Waterman kernels: 0x7c00 - bias - largest table entry
LIMIT_BLOSUM62 = 0x7c00 - 1024 - 11


def _expected(c, q):
    l8, l16 = lanes(c["simd"])
    cfg = oracle.SearchConfig(algo=c["algo"], bit_width=c["width"], align_type=c["align"], hitcount=c["hits"],
                              chunk_size=c["chunk"], gap_open=c["gap"][0], gap_extend=c["gap"][1], lanes8=l8,
                              lanes16=l16, matrix=c["table"])
    db = [oracle.map_codes(r.decode(), False, False) for r in c["records"]]
    res, ovf = oracle.search(cfg, oracle.map_codes(q.decode(), False, True), db)
    return [(h.id, h.score, h.cigar, h.q_start, h.q_end, h.d_start, h.d_end) for h in res], tuple(ovf)


def _check(c, scale=1):
    product_setup(1, ("builtin", "blosum62"), c["gap"], c["chunk"], c["simd"], records=c["records"])
    if scale != 1:
        import libssa_b200 as L
        # the BLOSUM62 text with every entry multiplied
        lines = open(os.path.join(DATA, "wide_scores.txt")).read().splitlines()
        base = 100000007
        text = "\n".join(ln if ln.startswith("#") else
                         " ".join(str(int(t) // base * scale) if t.lstrip("-").isdigit() else t for t in ln.split())
                         for ln in lines) + "\n"
        L.init_score_matrix(L.READ_FROM_STRING, text)
        c = dict(c, table=oracle.parse_matrix(text))
    else:
        c = dict(c, table=matrix_table(("builtin", "blosum62")))
    batched, _ = product_search(c["algo"], c["width"], c["align"], c["hits"], c["queries"], batch=True)
    single, ovf = product_search(c["algo"], c["width"], c["align"], c["hits"], c["queries"])
    for qi, q in enumerate(c["queries"]):
        exp, eovf = _expected(c, q)
        assert batched[qi] == exp, (qi, len(q))
        assert single[qi] == exp, (qi, len(q))
        assert tuple(ovf[qi]) == eovf, (qi, len(q))


@pytest.mark.parametrize("width", [16, 64])
def test_scores_around_the_16x2_range(built_library, width):
    """Runs of W score 11 per residue: the longest below the range, the first
    at it and past it, and (16 bits) past the lane's own 65535."""
    n = (LIMIT_BLOSUM62 + 10) // 11            # the first length that reaches the limit
    rng = np.random.default_rng(11)
    records = [b"W" * k for k in (n - 1, n, n + 1, n + 4, 5957, 5958, 5959)]
    records += [W.random_residues(rng, k, W.AA20).tobytes() for k in (1, 3, 4, 5, 127, 128, 129, 700)]
    _check(dict(algo="sw", width=width, align=0, hits=15, gap=(-11, -1), chunk=4, simd=2, records=records,
                queries=[b"W" * 5960, b"W" * n, b"W" * (n - 1)]))


@pytest.mark.parametrize("algo,width", [("sw", 16), ("sw", 64), ("nw", 64)])
@pytest.mark.parametrize("scale", [1, 16, 4000])
def test_score_tables_beyond_int8_and_int16(built_library, algo, width, scale):
    """BLOSUM62, 16 times it (entries past int8) and 4,000 times it (past
    int16 at 64 bits, truncated at 16)."""
    rng = np.random.default_rng(12 + scale)
    queries = [W.random_residues(rng, n, W.AA20) for n in (1, 80, 81, 333, 640)]
    records = [W.mutate(rng, q, W.AA20, 0.1, 0.02, (1, 4)).tobytes() for q in queries for _ in range(2)]
    records += [W.random_residues(rng, int(n), W.AA20).tobytes() for n in rng.integers(1, 900, 60)]
    records.append(W.random_residues(rng, 7001, W.AA20).tobytes())
    _check(dict(algo=algo, width=width, align=0, hits=12, gap=(-11, -1), chunk=50, simd=2, records=records,
                queries=[q.tobytes() for q in queries]), scale)


@pytest.mark.parametrize("width", [16, 64])
@pytest.mark.parametrize("gap", [(-11, -1), (-10, 0), (0, 0), (0, -2), (-128, -127), (3, -1)])
def test_gap_settings(built_library, width, gap):
    """Free, zero and extreme gap penalties; a positive opening stays with the
    lane emulation."""
    rng = np.random.default_rng(13)
    queries = [W.random_residues(rng, n, W.AA20) for n in (40, 257)]
    records = [W.mutate(rng, q, W.AA20, 0.1, 0.05, (1, 4)).tobytes() for q in queries for _ in range(3)]
    records += [W.random_residues(rng, int(n), W.AA20).tobytes() for n in rng.integers(1, 500, 40)]
    _check(dict(algo="sw", width=width, align=0, hits=10, gap=gap, chunk=1000, simd=1, records=records,
                queries=[q.tobytes() for q in queries]))
