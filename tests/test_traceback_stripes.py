"""Traceback passes on streamed stripes, 4 and 8 rows per lane: queries around
the stripe edges (128 and 256 rows), columns around the 32-column chunks, score
tables inside and past int8, symmetric and not, against the oracle: scores,
order, CIGARs and coordinates."""
import numpy as np
import pytest

import oracle
from helpers import product_search, product_setup
from libssa_b200 import workloads as W

pytestmark = pytest.mark.gpu

AA = "ARNDCQEGHILKMFPSTWYV"


def _matrix_text(scale: int, symmetric: bool, rng) -> str:
    m = rng.integers(-4, 3, (20, 20))
    m = np.tril(m) + np.tril(m, -1).T
    np.fill_diagonal(m, rng.integers(4, 9, 20))
    if not symmetric:
        m[3, 7], m[7, 3], m[0, 5] = 2, -3, 1
    return "\n".join(["  " + " ".join(AA)] + [AA[i] + " " + " ".join(str(int(v) * scale) for v in m[i])
                                              for i in range(20)]) + "\n"


@pytest.mark.parametrize("rows", [4, 8])
@pytest.mark.parametrize("algo,scale,symmetric", [("sw", 1, True), ("sw", 40, True), ("sw", 1, False), ("nw", 1, True),
                                                  ("nw", 40, False)])
def test_stripe_edges(built_library, monkeypatch, rows, algo, scale, symmetric):
    import libssa_b200 as L
    monkeypatch.setenv("SSA_B200_TB_R", str(rows))
    rng = np.random.default_rng(100 * scale + rows)
    text = _matrix_text(scale, symmetric, rng)
    table = oracle.parse_matrix(text)
    gap = (-11 * scale if scale == 1 else -120, -1 * scale)
    queries = [W.random_residues(rng, n, W.AA20) for n in (1, 4, 5, 127, 128, 129, 256, 257, 520)]
    records = [W.random_residues(rng, n, W.AA20) for n in (2, 3, 31, 32, 33, 63, 64, 65, 97, 300)]
    records += [W.mutate(rng, q, W.AA20, 0.15, 0.05, (1, 9)) for q in queries[3:]]
    records = [r.tobytes() for r in records]
    product_setup(1, ("builtin", "blosum62"), gap, 1000, 2, records=records)
    L.init_score_matrix(L.READ_FROM_STRING, text)
    queries = [q.tobytes() for q in queries]
    got, _ = product_search(algo, 64, 1, 12, queries, batch=True)
    db = [oracle.map_codes(r.decode(), False, False) for r in records]
    for qi, q in enumerate(queries):
        cfg = oracle.SearchConfig(algo=algo, bit_width=64, align_type=1, hitcount=12, chunk_size=1000,
                                  gap_open=gap[0], gap_extend=gap[1], lanes8=32, lanes16=16, matrix=table)
        res, _ = oracle.search(cfg, oracle.map_codes(q.decode(), False, True), db)
        exp = [(h.id, h.score, h.cigar, h.q_start, h.q_end, h.d_start, h.d_end) for h in res]
        assert got[qi] == exp, (qi, len(q))
