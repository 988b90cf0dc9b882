"""The searches that this library is measured on, through its Python entry points.

A case is one call (or one burst of calls) that a program makes while it holds a
database: ``sw_align`` / ``nw_align`` of one query, ``align_batch`` of many,
``align_pairs`` of long sequences against their partners, or a burst of requests
to a running ``Server``.  The database, the settings and a running server are
what such a program keeps from call to call, so they follow from the case alone;
the queries, which are new in every call, follow from the seed.

Sequences are random residues; about 1% of a database's records are relatives of
the case's queries, as a search in earnest meets them: mutated copies of the
query's family (70-95% identity), or, in a ``tiled`` database, copies repeated to
8,000-35,000 residues at 98% identity.  Lengths and settings are those of the
library's own workloads (libssa_b200/workloads.py): protein records gamma(2,
mean 350), nucleotide records U[100, 1500], queries lognormal around a median,
BLOSUM62 with gaps 11/1 or match 2 / mismatch -3 with gaps 5/2.

All outputs are whole numbers and bytes.
"""
from __future__ import annotations

import math
import statistics

import numpy as np
import torch

import libssa_b200 as L
from libssa_b200 import workloads as W

PROTEIN_GAPS, NUCLEOTIDE_GAPS = (-11, -1), (-5, -2)
MATCH, MISMATCH = 2, -3

# BLOSUM62 over the residues that the sequences hold (a published table)
BLOSUM62 = """
 4 -1 -2 -2  0 -1 -1  0 -2 -1 -1 -1 -1 -2 -1  1  0 -3 -2  0
-1  5  0 -2 -3  1  0 -2  0 -3 -2  2 -1 -3 -2 -1 -1 -3 -2 -3
-2  0  6  1 -3  0  0  0  1 -3 -3  0 -2 -3 -2  1  0 -4 -2 -3
-2 -2  1  6 -3  0  2 -1 -1 -3 -4 -1 -3 -3 -1  0 -1 -4 -3 -3
 0 -3 -3 -3  9 -3 -4 -3 -3 -1 -1 -3 -1 -2 -3 -1 -1 -2 -2 -1
-1  1  0  0 -3  5  2 -2  0 -3 -2  1  0 -3 -1  0 -1 -2 -1 -2
-1  0  0  2 -4  2  5 -2  0 -3 -3  1 -2 -3 -1  0 -1 -3 -2 -2
 0 -2  0 -1 -3 -2 -2  6 -2 -4 -4 -2 -3 -3 -2  0 -2 -2 -3 -3
-2  0  1 -1 -3  0  0 -2  8 -3 -3 -1 -2 -1 -2 -1 -2 -2  2 -3
-1 -3 -3 -3 -1 -3 -3 -4 -3  4  2 -3  1  0 -3 -2 -1 -3 -1  3
-1 -2 -3 -4 -1 -2 -3 -4 -3  2  4 -2  2  0 -3 -2 -1 -2 -1  1
-1  2  0 -1 -3  1  1 -2 -1 -3 -2  5 -1 -3 -1  0 -1 -3 -2 -2
-1 -1 -2 -3 -1  0 -2 -3 -2  1  2 -1  5  0 -2 -1 -1 -1 -1  1
-2 -3 -3 -3 -2 -3 -3 -3 -1  0  0 -3  0  6 -4 -2 -2  1  3 -1
-1 -2 -2 -1 -3 -1 -1 -2 -2 -3 -3 -1 -2 -4  7 -1 -1 -4 -3 -2
 1 -1  1  0 -1  0  0  0 -1 -2 -2  0 -1 -2 -1  4  1 -3 -2 -2
 0 -1  0 -1 -1 -1 -1 -2 -2 -1 -1 -1 -1 -2 -1  1  5 -2 -2  0
-3 -3 -4 -4 -2 -2 -3 -2 -2 -3 -2 -3 -1  1 -4 -3 -2 11  2 -3
-2 -2 -2 -3 -2 -1 -2 -3  2 -1 -1 -2 -1  3 -3 -2 -2  2  7 -1
 0 -3 -3 -3 -1 -2 -2 -3 -3  3  1 -2  1 -1 -2 -2  0 -3 -1  4
"""
BLOSUM62_ORDER = b"ARNDCQEGHILKMFPSTWYV"


def _case(name, kind, algo, width, align, hits, residues, queries, qlen, spread, records, tiled=False):
    """kind: single, batch, served or pairs; residues: protein, nucleotide, both_strands or translated (the query
    is nucleotides, the database protein); qlen, spread: median and lognormal sigma of the query lengths (for
    pairs: shortest and longest record)."""
    return {"name": name, "kind": kind, "algo": algo, "width": width, "align": align, "hits": hits,
            "residues": residues, "queries": queries, "qlen": qlen, "spread": spread, "records": records,
            "tiled": tiled}


def listed():
    return [
        # the smallest call: a peptide looked up among a few hundred proteins
        _case("sw_peptide_500", "single", "sw", 8, True, 5, "protein", 1, 40, 0.0, 500),
        # one protein against one proteome, the library's first workload
        _case("sw_protein_10k", "single", "sw", 8, True, 10, "protein", 1, 375, 0.0, 10_000),
        # one protein against a large database with very long relatives
        _case("sw_protein_tiled_200k", "single", "sw", 8, True, 10, "protein", 1, 300, 0.0, 200_000, True),
        # an ordinary batch: the proteins of one experiment against one proteome
        _case("sw_batch_32x20k", "batch", "sw", 8, True, 10, "protein", 32, 300, 0.7, 20_000),
        # the largest call: annotation of many proteins against a large database
        _case("sw_batch_96x200k", "batch", "sw", 8, True, 10, "protein", 96, 300, 0.7, 200_000, True),
        # the 16-bit entry, which callers with close relatives choose (no 8-bit pass to repeat)
        _case("sw16_batch_24x20k", "batch", "sw", 16, True, 10, "protein", 24, 300, 0.7, 20_000),
        # the exact 64-bit entry, scores alone
        _case("sw64_protein_10k", "single", "sw", 64, False, 10, "protein", 1, 375, 0.0, 10_000),
        # global alignment of reads against a reference collection, 16-bit entry
        _case("nw16_nucleotide_64x20k", "batch", "nw", 16, True, 20, "nucleotide", 64, 340, 0.4, 20_000),
        # global alignment through the whole cascade, the library's default width
        _case("nw8_protein_20k", "single", "nw", 8, True, 10, "protein", 1, 250, 0.0, 20_000),
        # a read whose strand is unknown
        _case("sw_both_strands_50k", "single", "sw", 8, True, 10, "both_strands", 1, 500, 0.0, 50_000),
        # long proteins against their partners, local and global
        _case("pairs_48", "pairs", "both", 16, True, 1, "protein", 48, 5000, 30000.0, 48),
        # a burst of requests to a running server
        _case("served_32x100k", "served", "sw", 8, True, 10, "protein", 32, 300, 0.8, 100_000),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the listed ones' ranges; its cells stay below what its kind computes in about the time of the
    largest listed case."""
    kind = rng.choice(["single", "single", "batch", "batch", "served", "pairs"])
    if kind == "pairs":
        n, lo = _log_uniform(rng, 2, 64), rng.randint(3000, 8000)
        return _drop_name(_case("", "pairs", "both", 16, rng.random() < 0.8, 1, "protein", n, lo,
                                float(rng.randint(lo + 1000, 30000)), n))
    algo = "sw" if kind == "served" else rng.choice(["sw", "sw", "nw"])
    width = 8 if kind == "served" else rng.choice([8, 8, 16, 64] if algo == "sw" else [8, 16, 16, 64])
    residues = "protein"
    if kind != "served":
        residues = rng.choice(["protein", "protein", "protein", "nucleotide", "both_strands", "translated"])
    queries = 1 if kind == "single" else _log_uniform(rng, 2, 96)
    qlen = _log_uniform(rng, 30, 2000 if kind == "single" else 600)
    spread = 0.0 if kind == "single" else round(rng.uniform(0.2, 0.8), 2)
    tiled = residues == "protein" and algo == "sw" and width == 8 and rng.random() < 0.3
    most = 2e12 if algo == "sw" and width == 8 else 1.5e11
    per_record = {"protein": 700 if tiled else 350, "translated": 6 * 350 / 3, "nucleotide": 800,
                  "both_strands": 4 * 800}[residues]
    records = min(_log_uniform(rng, 150, 200_000), int(most / (queries * 1.4 * qlen * per_record)))
    return _drop_name(_case("", kind, algo, width, rng.random() < 0.7, rng.choice([1, 5, 10, 20, 50]), residues, queries,
                            qlen, spread, max(100, records), tiled))


def _drop_name(case):
    del case["name"]
    return case


def _lengths(case):
    """The query lengths: evenly spaced quantiles, so that every seed's queries cost the same."""
    n = case["queries"]
    if case["kind"] == "pairs":
        return [int(case["qlen"] + (case["spread"] - case["qlen"]) * (i + 0.5) / n) for i in range(n)]
    normal = statistics.NormalDist()
    out = [case["qlen"] * math.exp(case["spread"] * normal.inv_cdf((i + 0.5) / n)) for i in range(n)]
    lens = [min(5000, max(30, int(round(x)))) for x in out]
    return [3 * (x // 3) + 30 for x in lens] if case["residues"] == "translated" else lens


def _alphabet(case):
    return W.NT4 if case["residues"] in ("nucleotide", "both_strands") else W.AA20


def _families(case):
    """One ancestor per query; the database's relatives and the queries descend from it."""
    rng = np.random.default_rng([case["queries"], case["qlen"], case["records"], 1])
    alphabet = W.NT4 if case["residues"] == "translated" else _alphabet(case)
    return [W.random_residues(rng, n, alphabet) for n in _lengths(case)]


def _database(case):
    """The case's database: residues back to back and record offsets."""
    families = _families(case)
    if case["kind"] == "pairs":
        records = families
    else:
        rng = np.random.default_rng([case["queries"], case["qlen"], case["records"], 2])
        alphabet, n = _alphabet(case), case["records"]
        if alphabet is W.NT4:
            lens = rng.integers(100, 1501, n)
        else:
            lens = W.gamma_lengths(rng, n, 350.0, 20, 35000 if case["tiled"] else 5000)
        bulk = W.random_residues(rng, int(lens.sum()), alphabet)
        records = np.split(bulk, np.cumsum(lens)[:-1])
        for i in np.flatnonzero(rng.random(n) < 0.01):
            source = families[int(rng.integers(0, len(families)))]
            if case["residues"] == "translated":
                continue            # a translated query's relatives are those that its frames happen to meet
            if case["tiled"]:
                target = int(rng.integers(8000, 35001))
                records[i] = W.mutate(rng, np.tile(source, target // len(source) + 1)[:target], alphabet, 0.02, 0.0, (1, 1))
            else:
                records[i] = W.mutate(rng, source, alphabet, rng.uniform(0.05, 0.30), 0.01, (1, 5))
    offsets = np.zeros(len(records) + 1, dtype=np.uint64)
    offsets[1:] = np.cumsum([len(r) for r in records])
    return np.concatenate(records).astype(np.uint8), offsets


def _queries(case, seed):
    """The call's queries: each 5% (a pair's: 1-15%, with insertions and deletions) from its ancestor."""
    rng = np.random.default_rng([seed, 3])
    alphabet = W.NT4 if case["residues"] == "translated" else _alphabet(case)
    if case["kind"] == "pairs":
        return [W.mutate(rng, f, alphabet, rng.uniform(0.01, 0.15), 0.01, (1, 20)) for f in _families(case)]
    return [W.mutate(rng, f, alphabet, 0.05, 0.0, (1, 1)) for f in _families(case)]


class _Session:
    """What the program holds between calls: the loaded database, the settings and, for served cases, the server.
    The library keeps one database per process, so a session ends when another case's begins."""

    current = None

    @classmethod
    def of(cls, case):
        key = {k: v for k, v in case.items() if k != "name"}
        if cls.current is None or cls.current.key != key:
            if cls.current is not None and cls.current.server is not None:
                cls.current.server.stop()
            cls.current = cls(case, key)
        return cls.current

    def __init__(self, case, key):
        self.key, self.server = key, None
        L.set_output_mode(L.OUTPUT_SILENT)
        symbols = {"protein": L.AMINOACID, "translated": L.TRANS_QUERY}.get(case["residues"], L.NUCLEOTIDE)
        both = case["residues"] in ("both_strands", "translated")
        L.init_symbol_translation(symbols, L.BOTH_STRANDS if both else L.FORWARD_STRAND, 1, 1)
        if symbols == L.NUCLEOTIDE:
            L.init_constant_scores(MATCH, MISMATCH)
            L.init_gap_penalties(*NUCLEOTIDE_GAPS)
        else:
            L.init_score_matrix(L.MATRIX_BUILDIN, "blosum62")
            L.init_gap_penalties(*PROTEIN_GAPS)
        L.set_chunk_size(1000)
        L.set_simd_compute_mode(L.COMPUTE_ON_AVX2)
        L.set_thread_count(1)
        flat, offsets = _database(case)
        L.load_db_memory(flat=flat, offsets=offsets)
        if case["kind"] == "served":
            self.server = L.Server(L.SSA_SMITH_WATERMAN, case["hits"], case["width"], _align(case))


class _Call:
    """One call's state: its query handles, given back with it."""

    def __init__(self, case, seed):
        self.case, self.session, self.lengths = case, _Session.of(case), _lengths(case)
        self.queries = [L.init_sequence_fasta(L.READ_FROM_STRING, q.tobytes().decode()) for q in _queries(case, seed)]

    def __del__(self):
        for q in self.queries:
            L.free_sequence(q)


def _align(case):
    return L.COMPUTE_ALIGNMENT if case["align"] else L.COMPUTE_SCORE


def prepare(case, seed):
    return _Call(case, seed)


def run(state):
    case, queries = state.case, state.queries
    algo = L.SSA_NEEDLEMAN_WUNSCH if case["algo"] == "nw" else L.SSA_SMITH_WATERMAN
    if case["kind"] == "single":
        align = L.nw_align if case["algo"] == "nw" else L.sw_align
        lists = [align(queries[0], case["hits"], case["width"], _align(case))]
    elif case["kind"] == "batch":
        lists = L.align_batch(algo, queries, case["hits"], case["width"], _align(case))
    elif case["kind"] == "served":
        tickets = [state.session.server.submit(q) for q in queries]
        lists = [state.session.server.wait(t)[0] for t in tickets]
    else:
        ids = list(range(len(queries)))
        lists = [hits for a in (L.SSA_SMITH_WATERMAN, L.SSA_NEEDLEMAN_WUNSCH)
                 for hits in L.align_pairs(a, queries, ids, case["width"], _align(case))]
    hits = [h for found in lists for h in found]
    # one zero-filled text of a fixed length per list: a query of n residues gives at most 8 n + 6 characters per hit
    # (n runs of matches or insertions, at most n + 1 deletion runs of up to 6 characters between them); a quarter more
    # for a pair's query, which its mutation may have made longer
    lengths = state.lengths * (len(lists) // len(queries))
    cigars = np.zeros(case["hits"] * sum(8 * (n + n // 4 + 32) for n in lengths) if case["align"] else 0, dtype=np.uint8)
    text = np.frombuffer("\n".join(h.cigar or "" for h in hits).encode()[:len(cigars)], dtype=np.uint8)
    cigars[:len(text)] = text
    return {"count": np.array([len(found) for found in lists], dtype=np.int64),
            "score": np.array([h.score for h in hits], dtype=np.int64),
            "where": np.array([(h.id, h.q_start, h.q_end, h.d_start, h.d_end, h.strand, h.frame, h.qstrand, h.qframe)
                               for h in hits], dtype=np.int64),
            "cigar": cigars}


def _residues(case):
    """Residues of the case's database, without making it where its lengths are known."""
    if case["kind"] == "pairs":
        return sum(_lengths(case))
    if _alphabet(case) is W.NT4:
        return case["records"] * 800
    return case["records"] * (350 + (215 if case["tiled"] else 0))


def _cells(case):
    """Cells of the dynamic-programming matrices that the call asks for."""
    lens = _lengths(case)
    if case["kind"] == "pairs":
        return 2 * sum(n * n for n in lens)             # local and global
    # strands: 2 of the query against 2 of the database; frames: 6 of a third of the length
    return sum(lens) * _residues(case) * {"both_strands": 4, "translated": 2}.get(case["residues"], 1)


def work(case):
    """The database and the queries read once, the hits written once; 4 additions and 5 maxima per cell."""
    hits = min(case["hits"], case["records"]) * case["queries"]
    return {"bytes": float(_residues(case) + sum(_lengths(case)) + 96 * hits), "flops": 9.0 * _cells(case)}


# ---- plain 64-bit scores --------------------------------------------------------------
def _codes(case, seqs):
    order = BLOSUM62_ORDER if _alphabet(case) is W.AA20 else b"ACGT"
    table = np.full(256, -1, dtype=np.int64)
    table[np.frombuffer(order, dtype=np.uint8)] = np.arange(len(order))
    return [table[s] for s in seqs]


def _scores(case, query, records):
    """Exact scores of one query against all records: one anti-diagonal of all matrices at a time."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if _alphabet(case) is W.AA20:
        table, (go, ge) = torch.tensor([[int(x) for x in row.split()] for row in BLOSUM62.strip().splitlines()]), PROTEIN_GAPS
    else:
        table, (go, ge) = torch.full((4, 4), MISMATCH) + torch.eye(4, dtype=torch.int64) * (MATCH - MISMATCH), NUCLEOTIDE_GAPS
    local = case["algo"] == "sw"
    lens = torch.tensor([len(r) for r in records], device=dev)
    n, q, width = len(records), len(query), int(lens.max())
    # the records reversed and padded with -1 on both sides: an anti-diagonal is then a window of q columns
    padded = np.full((n, q + width + q), -1, dtype=np.int64)
    for i, r in enumerate(records):
        padded[i, q + width - len(r):q + width] = r[::-1]
    padded = torch.from_numpy(padded).to(dev)
    scores_of = torch.cat([table.to(dev)[torch.from_numpy(query).to(dev)], torch.full((q, 1), -1000, device=dev)], 1)
    rows = torch.arange(q, device=dev)
    low = -(1 << 40)
    start = torch.zeros(q + 1, dtype=torch.int64, device=dev) if local else torch.cat(
        [torch.zeros(1, dtype=torch.int64, device=dev), go + (rows + 1) * ge])
    h1 = torch.full((n, q + 1), low, device=dev)            # H of the last anti-diagonal, a row above the first included
    h2 = h1.clone()
    e, f = torch.full((n, q), low, device=dev), torch.full((n, q), low, device=dev)
    best = torch.zeros(n, dtype=torch.int64, device=dev)
    h1[:, 0] = 0
    for d in range(q + width - 1):
        # cell (i, j = d - i); h1[:, i + 1] is H(i, j - 1), h1[:, i] is H(i - 1, j), h2[:, i] is H(i - 1, j - 1)
        if d < q:                                           # row d enters at column 0: its left and diagonal neighbours
            h1[:, d + 1] = start[d + 1]
            h2[:, d] = start[d]
            e[:, d] = start[d + 1] + go if not local else low
        h1[:, 0] = 0 if local else go + (d + 1) * ge        # above row 0 in column d
        h2[:, 0] = 0 if local or d == 0 else go + d * ge
        e = torch.maximum(e + ge, h1[:, 1:] + go + ge)
        f_above = torch.cat([torch.full((n, 1), low, device=dev), f[:, :-1]], 1)
        f = torch.maximum(f_above + ge, h1[:, :-1] + go + ge)
        at = q + width - 1 - d + rows                       # column of record residue d - i in the reversed layout
        code = padded[:, at.clamp(0, padded.shape[1] - 1)]
        column = lens - 1                                   # records end at their own last column
        h = torch.maximum(torch.maximum(e, f), h2[:, :-1] + scores_of[rows, code])
        inside = (d - rows >= 0)[None, :] & ((d - rows)[None, :] <= column[:, None])
        if local:
            h = h.clamp(min=0)
            best = torch.maximum(best, torch.where(inside, h, torch.zeros_like(h)).amax(1))
        else:
            best = torch.where(column == d - (q - 1), h[:, -1], best)
        h2 = h1
        h1 = torch.cat([h1[:, :1], h], 1)
    return best


def exact(case, seed):
    """The hits' scores, which no tie can change; the rest of a call's outputs follows from its search order."""
    if case["kind"] not in ("single", "batch") or case["residues"] not in ("protein", "nucleotide") or case["tiled"] \
            or _cells(case) > 4e9:
        return None
    flat, offsets = _database(case)
    records = _codes(case, [flat[int(a):int(b)] for a, b in zip(offsets, offsets[1:])])
    found = [torch.sort(_scores(case, q, records), descending=True).values[:case["hits"]]
             for q in _codes(case, _queries(case, seed))]
    return {"count": np.array([len(s) for s in found], dtype=np.int64), "score": torch.cat(found).cpu().numpy(),
            "where": None, "cigar": None}
