"""Score tables past int8 and past int16 (BLOSUM62 with every entry multiplied)
at every entry width: which kernels may take them, the 16-bit pass after the
8-bit entry, sequences around the 16x2 range, and the traceback.  Hits, order,
CIGARs, coordinates and overflow counters against the oracle."""
import os

import numpy as np
import pytest

import oracle
from helpers import DATA, product_search, product_setup
from libssa_b200 import workloads as W
from test_wide_entry import _expected


def scaled_blosum62(scale):
    """The table's text, entries of 100,000,007 x BLOSUM62 brought to scale x BLOSUM62."""
    out = []
    for ln in open(os.path.join(DATA, "wide_scores.txt")).read().splitlines():
        if not ln.startswith("#"):
            ln = ("   " if ln[0] == " " else "") + " ".join(
                str(round(int(t) / 100000007) * scale) if t.lstrip("-").isdigit() else t for t in ln.split())
        out.append(ln)
    return "\n".join(out) + "\n"


def check_scaled(c, scale):
    import libssa_b200 as L
    text = scaled_blosum62(scale)
    c = dict(c, table=oracle.parse_matrix(text), records=[r.tobytes() for r in c["records"]],
             queries=[q.tobytes() for q in c["queries"]])
    product_setup(1, ("builtin", "blosum62"), c["gap"], c["chunk"], c["simd"], records=c["records"])
    L.init_score_matrix(L.READ_FROM_STRING, text)
    batched, _ = product_search(c["algo"], c["width"], c["align"], c["hits"], c["queries"], batch=True)
    single, ovf = product_search(c["algo"], c["width"], c["align"], c["hits"], c["queries"])
    for qi, q in enumerate(c["queries"]):
        exp, eovf = _expected(c, q)
        assert batched[qi] == exp, (qi, len(q))
        assert single[qi] == exp, (qi, len(q))
        assert tuple(ovf[qi]) == eovf, (qi, len(q))


def test_the_scaled_text_is_the_table_multiplied():
    one = oracle.parse_matrix(scaled_blosum62(1))
    assert one.max() == 11 and one.min() == -4
    for scale in (16, 4000):
        t = oracle.parse_matrix(scaled_blosum62(scale))
        assert t.max() == 11 * scale and (t[one > 0] == scale * one[one > 0]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("algo", ["sw", "nw"])
@pytest.mark.parametrize("width", [8, 16, 64])
@pytest.mark.parametrize("scale", [1, 11, 16, 700, 4000])
def test_scaled_tables(built_library, algo, width, scale):
    """11: the largest table within int8; 16: past it; 700: SW entries up to
    7,700, under the 8,192 that the 16x2 kernels take; 4000: past int16."""
    rng = np.random.default_rng(80 + scale)
    queries = [W.random_residues(rng, n, W.AA20) for n in (3, 50, 129, 300)]
    records = [W.mutate(rng, q, W.AA20, rate, 0.02, (1, 3)) for q in queries for rate in (0.0, 0.1, 0.4)]
    records += [W.random_residues(rng, int(n), W.AA20) for n in rng.integers(1, 400, 40)]
    check_scaled(dict(algo=algo, width=width, align=1, hits=14, gap=(-11, -1), chunk=20, simd=2, records=records,
                      queries=queries), scale)
