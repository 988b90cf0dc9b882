"""Traceback passes on streamed stripes: queries around the stripe edges (128 and
256 rows), columns around the 4-column blocks and 16-block chunks, score
tables inside and past int8, symmetric and not, against the oracle: scores,
order, CIGARs and coordinates."""
import numpy as np
import pytest

import oracle
from helpers import matrix_table, product_search, product_setup
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


@pytest.mark.parametrize("algo,scale,symmetric", [("sw", 1, True), ("sw", 40, True), ("sw", 1, False), ("nw", 1, True),
                                                  ("nw", 40, False)])
def test_stripe_edges(built_library, algo, scale, symmetric):
    import libssa_b200 as L
    rng = np.random.default_rng(100 * scale + 4)
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


@pytest.mark.parametrize("algo", ["sw", "nw"])
def test_pair_scores(built_library, algo):
    """Scores of pairs without alignments on the same sweep."""
    import libssa_b200 as L
    rng = np.random.default_rng(7)
    records = [W.random_residues(rng, n, W.AA20) for n in (1, 2, 3, 4, 5, 63, 64, 65, 127, 130, 700, 2500)]
    queries = [W.mutate(rng, np.tile(r, 2), W.AA20, 0.2, 0.05, (1, 4)) for r in records]
    queries = [q if len(q) else records[5] for q in queries]
    product_setup(1, ("builtin", "blosum62"), (-11, -1), 1000, 2, records=[r.tobytes() for r in records])
    qs = [L.init_sequence_fasta(L.READ_FROM_STRING, q.tobytes().decode()) for q in queries]
    got = L.align_pairs(L.SSA_SMITH_WATERMAN if algo == "sw" else L.SSA_NEEDLEMAN_WUNSCH, qs, list(range(len(qs))), 16,
                        L.COMPUTE_SCORE)
    for q in qs:
        L.free_sequence(q)
    for i, (q, r) in enumerate(zip(queries, records)):
        cfg = oracle.SearchConfig(algo=algo, bit_width=64, align_type=0, hitcount=1, chunk_size=1000, gap_open=-11,
                                  gap_extend=-1, lanes8=32, lanes16=16, matrix=matrix_table(("builtin", "blosum62")))
        res, _ = oracle.search(cfg, oracle.map_codes(q.tobytes().decode(), False, True),
                               [oracle.map_codes(r.tobytes().decode(), False, False)])
        assert [h.score for h in got[i]] == [h.score for h in res], (i, len(q), len(r))


@pytest.mark.parametrize("gap", [(-11, -1), (0, -3)])
def test_two_rows_per_lane(built_library, monkeypatch, gap):
    """Stripes of 64 rows, which the library takes for a few hits much longer
    than they are high: queries around one, two and three of them."""
    monkeypatch.setenv("SSA_B200_TB_ROWS", "2")
    import libssa_b200 as L
    rng = np.random.default_rng(12)
    text = _matrix_text(1, True, rng)
    table = oracle.parse_matrix(text)
    queries = [W.random_residues(rng, n, W.AA20) for n in (1, 2, 3, 5, 63, 64, 65, 128, 129, 191, 260)]
    records = [W.random_residues(rng, n, W.AA20) for n in (61, 64, 65, 68, 129, 700)]
    records += [W.mutate(rng, np.tile(q, 2), W.AA20, 0.15, 0.05, (1, 9)) for q in queries[4:]]
    records = [r.tobytes() for r in records]
    product_setup(1, ("builtin", "blosum62"), gap, 1000, 2, records=records)
    L.init_score_matrix(L.READ_FROM_STRING, text)
    queries = [q.tobytes() for q in queries]
    got, _ = product_search("sw", 64, 1, 12, queries, batch=True)
    db = [oracle.map_codes(r.decode(), False, False) for r in records]
    for qi, q in enumerate(queries):
        cfg = oracle.SearchConfig(algo="sw", bit_width=64, align_type=1, hitcount=12, chunk_size=1000,
                                  gap_open=gap[0], gap_extend=gap[1], lanes8=32, lanes16=16, matrix=table)
        res, _ = oracle.search(cfg, oracle.map_codes(q.decode(), False, True), db)
        exp = [(h.id, h.score, h.cigar, h.q_start, h.q_end, h.d_start, h.d_end) for h in res]
        assert got[qi] == exp, (qi, len(q))
