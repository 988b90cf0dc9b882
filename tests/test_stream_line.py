"""Which calls stream the longest pairs of their entry pass: those whose few
longest pairs outlast the rest, and not those where streaming costs more than the
entry kernel takes for the same pairs (short queries, short records, flat
length distributions)."""
import re

import numpy as np
import pytest

from libssa_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _streamed(capfd, monkeypatch, algo, width, residues, lens, qlens):
    import libssa_b200 as L
    rng = np.random.default_rng(91)
    alphabet = W.AA20 if residues == "protein" else W.NT4
    flat = W.random_residues(rng, int(lens.sum()), alphabet)
    offsets = np.zeros(len(lens) + 1, dtype=np.uint64)
    offsets[1:] = np.cumsum(lens)
    L.set_output_mode(L.OUTPUT_SILENT)
    L.init_symbol_translation(L.AMINOACID if residues == "protein" else L.NUCLEOTIDE, L.FORWARD_STRAND, 1, 1)
    if residues == "protein":
        L.init_score_matrix(L.MATRIX_BUILDIN, "blosum62")
    else:
        L.init_constant_scores(2, -3)
    L.init_gap_penalties(-11, -1)
    L.set_chunk_size(1000)
    L.set_simd_compute_mode(L.COMPUTE_ON_AVX2)
    L.load_db_memory(flat=flat, offsets=offsets)
    queries = [L.init_sequence_fasta(L.READ_FROM_STRING, W.random_residues(rng, n, alphabet).tobytes().decode())
               for n in qlens]
    monkeypatch.setenv("SSA_B200_TIMING", "1")
    capfd.readouterr()
    try:
        L.align_batch(L.SSA_NEEDLEMAN_WUNSCH if algo == "nw" else L.SSA_SMITH_WATERMAN, queries, 5, width,
                      L.COMPUTE_SCORE)
    finally:
        for q in queries:
            L.free_sequence(q)
    found = re.findall(r"entry pass: (\d+) items streamed", capfd.readouterr().err)
    return [int(n) for n in found]


def _proteins(n, longest=5000):
    return W.gamma_lengths(np.random.default_rng(n), n, 350.0, 20, longest)


def _flat(n, lo, hi):
    return np.random.default_rng(n).integers(lo, hi + 1, n)


@pytest.mark.parametrize("algo,width,residues,lens,qlens,streams", [
    ("sw", 8, "nucleotide", _flat(20000, 100, 1500), [30], False),
    ("sw", 8, "nucleotide", _flat(20000, 100, 1500), [30, 28], False),
    ("nw", 16, "nucleotide", _flat(20000, 80, 150), [30], False),
    ("nw", 16, "nucleotide", _flat(100000, 80, 150), [100], False),
    ("nw", 16, "nucleotide", _flat(50000, 100, 1500), [80], False),
    ("sw", 8, "protein", _proteins(1500), [800], True),
    ("sw", 16, "protein", _proteins(1000), [150, 120, 110, 90], True),
    ("nw", 16, "protein", _proteins(5000), [300], True),
    ("nw", 64, "nucleotide", _flat(1500, 100, 1500), [800], True),
    ("sw", 8, "protein", np.concatenate([_proteins(20000), _flat(100, 8000, 35000)]), [300], True),
])
def test_where_streaming_pays(built_library, capfd, monkeypatch, algo, width, residues, lens, qlens, streams):
    found = _streamed(capfd, monkeypatch, algo, width, residues, lens, qlens)
    assert found and all((n > 0) == streams for n in found), found
