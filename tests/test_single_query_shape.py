"""The entry shape of single queries on databases of 30,000 to 50,000 records,
which may be that of the large-database costs: only where every group of threads
has work, else the small database's."""
import os

import numpy as np
import pytest

from libssa_b200 import workloads as W

pytestmark = pytest.mark.gpu

TABLE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "libssa_b200", "tuning", "b200.tune")


def _cheapest(bucket, q):
    """(G, R) of the least passes x cost among the table's single-query shapes."""
    best = {}
    for line in open(TABLE):
        f = line.split()
        if f and f[0] in ("fast", "fast4") and int(f[1]) == bucket:
            G, R = int(f[2]), int(f[3])
            best[f[0] == "fast4", G, R] = -(-q // (G * R)) * float(f[4])
    return min(best, key=best.get)[1:]


@pytest.mark.parametrize("records", [30000, 38000, 49999])
def test_shape(built_library, records):
    import libssa_b200 as L
    sms = 148
    rng = np.random.default_rng(92)
    lens = W.gamma_lengths(rng, records, 350.0, 20, 5000)
    flat = W.random_residues(rng, int(lens.sum()), W.AA20)
    offsets = np.zeros(records + 1, dtype=np.uint64)
    offsets[1:] = np.cumsum(lens)
    L.set_output_mode(L.OUTPUT_SILENT)
    L.init_symbol_translation(L.AMINOACID, L.FORWARD_STRAND, 1, 1)
    L.init_score_matrix(L.MATRIX_BUILDIN, "blosum62")
    L.init_gap_penalties(-11, -1)
    L.set_chunk_size(1000)
    L.set_simd_compute_mode(L.COMPUTE_ON_AVX2)
    L.load_db_memory(flat=flat, offsets=offsets)
    for q in (30, 80, 96, 150, 300, 800):
        handle = L.init_sequence_fasta(L.READ_FROM_STRING, W.random_residues(rng, q, W.AA20).tobytes().decode())
        L.sw_align(handle, 5, 8, L.COMPUTE_SCORE)
        L.free_sequence(handle)
        used = L.tuning_report()["last_call"][0]
        G, R = _cheapest(4, q)
        groups, passes = sms * 16 * (32 // G), -(-q // (G * R))
        crowded = 4 * ((records + 1) // 2) * passes >= 5 * groups
        assert (used["G"], used["R"]) == ((G, R) if crowded else _cheapest(1, q)), (q, used)
        assert used["bucket"] == 1
