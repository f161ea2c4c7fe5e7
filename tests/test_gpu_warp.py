"""The one-launch classification of short fragments against the oracle, at
the lengths where a lane's positions, a warp's pass, the packed window and
the entry list begin and end, and with more taxa per fragment than lanes or
map slots."""
import os

import numpy as np
import pytest

import kraken2_gb300 as k2g
import oracle
from gpu_util import classify_batch, to_dev, torch
from kraken_io import Batch

pytestmark = pytest.mark.gpu

K, L = 35, 31
MASK, TOGGLE = 0x3ffffffff3333333, 0xe37e28c4271b5a2d
ACGT = np.frombuffer(b"ACGT", np.uint8)
# around: k; 8 positions a lane; 32 lanes a pass; the 352 entries; the packed window
EDGES = [0, 1, 30, 31, 34, 35, 36, 38, 39, 42, 43, 46, 47, 62, 63, 100, 150, 151, 250, 286, 287, 294,
         295, 301, 534, 535, 1100, 2032, 2047, 2048, 2049, 2100, 4095, 4096, 4097, 8192, 20_000]
CUT = 4096    # single fragments from here on are cut into pieces (not in quick mode)

_cache = {}


def database(wide: bool, many: bool):
    """A table over a 120 kb genome: taxa in stretches of 60 to 2,000 k-mers,
    or (many) a taxon of its own for every k-mer.  Returns (db, genome, oracle)."""
    if (wide, many) in _cache:
        return _cache[wide, many]
    t = torch()
    rng = np.random.default_rng(17)
    genome = ACGT[rng.integers(0, 4, 120_000)]
    genome[50_000:50_400] = ord("A")          # low complexity
    genome[60_000:60_500] = np.tile(np.frombuffer(b"ACG", np.uint8), 167)[:500]
    nodes = 4000
    parent = np.zeros(nodes, np.uint64)
    parent[2:] = (rng.random(nodes - 2) * np.minimum(np.arange(1, nodes - 1), 300)).astype(np.uint64) + 1
    vb = 12
    db = k2g.Database.create(k2g.IndexOptions(K, L, MASK, TOGGLE, 1, 1, 0), 200_003,
                             (40 if wide else 32) - vb, vb, parent)
    d_seq = to_dev(np.concatenate([genome, np.zeros(16, np.uint8)]))
    off = to_dev(np.array([0, len(genome)], np.uint64))
    mins = t.zeros(len(genome), dtype=t.int64, device="cuda")
    amb = t.zeros(len(genome), dtype=t.uint8, device="cuda")
    st = t.cuda.current_stream().cuda_stream
    db.scan(d_seq.data_ptr(), off.data_ptr(), 1, mins.data_ptr(), amb.data_ptr(), st)
    n = len(genome) - K + 1
    if many:
        taxa = rng.integers(1, nodes, n).astype(np.int32)
    else:
        taxa = np.repeat(rng.integers(1, nodes, n), rng.integers(60, 2000, n))[:n].astype(np.int32)
        taxa[rng.random(n) < 0.3] = 0         # stretches of the genome that are not in the table
    d_tax = to_dev(taxa.view(np.uint32))
    db.build_insert(mins.data_ptr(), d_tax.data_ptr(), n, True, st)
    cells, _ = db.download()
    inf = db.info()
    o = oracle.Oracle(cells, inf.capacity, inf.key_bits, inf.value_bits, parent,
                      oracle.index_opts(K, L, MASK, TOGGLE))
    _cache[wide, many] = (db, genome, o)
    return _cache[wide, many]


def batch(genome, lens, seed, quals=False):
    rng = np.random.default_rng(seed)
    seqs = []
    for i, n in enumerate(lens):
        at = int(rng.integers(0, len(genome) - n + 1))
        s = genome[at:at + n].copy()
        if i % 5 == 1 and n:                  # substitutions
            s[rng.integers(0, n, max(1, n // 60))] = ACGT[rng.integers(0, 4, max(1, n // 60))]
        if i % 7 == 2 and n > 3:              # ambiguous bases: alone, in runs, at the ends
            for p in rng.integers(0, n, 1 + n // 90):
                s[p:p + int(rng.integers(1, 45))] = ord("N")
            s[0] = ord("n")
            s[-1] = ord("N")
        if i % 11 == 3:
            s = np.frombuffer(bytes(s).lower(), np.uint8)
        if i % 13 == 4:
            s = ACGT[rng.integers(0, 4, n)]
        seqs.append(bytes(s))
    bases = b"".join(seqs)
    q = rng.integers(33, 74, len(bases)).astype(np.uint8).tobytes() if quals else None
    off = np.concatenate([[0], np.cumsum([len(x) for x in seqs])]).astype(np.uint64)
    return bases, q, off


def check(db, o, bases, q, off, n, params, mode=k2g.MODE_PIPELINED):
    b = Batch(bases, q, off, n, params.get("paired", False), [""] * n, [(0,)] * n, np.zeros(n, np.uint32))
    r = classify_batch(db, b, params, mode=mode)
    assert r.status == 0
    calls, hg, nr, runs, base = o.classify(bases, q, off, n, threads=os.cpu_count() or 1, **params)
    assert np.array_equal(r.call[:n], calls.astype(np.uint32))
    assert np.array_equal(r.hit_groups[:n], hg.astype(np.uint32))
    nr = nr.astype(np.int64)
    assert np.array_equal(r.hitlist_len[:n], nr)
    idx = np.repeat(r.hitlist_off[:n].astype(np.int64), nr) + \
        (np.arange(int(nr.sum())) - np.repeat(np.cumsum(nr) - nr, nr))
    odx = np.repeat(base.astype(np.int64), nr) + \
        (np.arange(int(nr.sum())) - np.repeat(np.cumsum(nr) - nr, nr))
    got, want = r.runs[idx], runs[odx]
    assert np.array_equal(got >> np.uint64(32), want["code"].astype(np.uint64) & np.uint64(0xFFFFFFFF))
    assert np.array_equal(got & np.uint64(0xFFFFFFFF), want["count"].astype(np.uint64))
    # nothing is written outside the runs of fragments that stay whole
    untouched = np.ones(len(r.runs), bool)
    untouched[idx] = False
    if not params.get("paired") and not params.get("quick"):
        for f in np.flatnonzero(np.diff(off.astype(np.int64)) >= CUT):
            untouched[int(off[f]) + 2 * f:int(off[f + 1]) + 2 * f + 2] = False
    assert not r.runs[untouched].any()
    assert np.array_equal(r.taxon_reads, np.bincount(calls[calls > 0].astype(np.int64), minlength=len(r.taxon_reads)))


PARAMS = [dict(confidence=0.0, min_hit_groups=0), dict(confidence=0.15, min_hit_groups=2),
          dict(confidence=0.0, min_hit_groups=2, min_quality=12), dict(confidence=0.0, min_hit_groups=3, quick=True),
          dict(confidence=0.6, min_hit_groups=1, paired=True),
          dict(confidence=0.0, min_hit_groups=2, paired=True, quick=True, min_quality=5)]


@pytest.mark.parametrize("many", [False, True], ids=["stretches", "taxon_per_kmer"])
@pytest.mark.parametrize("wide", [False, True], ids=["cells32", "cells40"])
@pytest.mark.parametrize("params", PARAMS, ids=lambda p: "-".join(f"{k}{v}" for k, v in p.items()))
def test_edge_lengths_equal_the_oracle(params, wide, many):
    db, genome, o = database(wide, many)
    rng = np.random.default_rng(5)
    lens = EDGES + [int(x) for x in rng.permutation(EDGES)] + [int(x) for x in rng.integers(0, 400, 300)]
    if params.get("paired"):
        lens = lens[:len(lens) // 2 * 2]
    bases, q, off = batch(genome, lens, 6, "min_quality" in params)
    check(db, o, bases, q, off, len(lens) // (2 if params.get("paired") else 1), params)


@pytest.mark.parametrize("n,hi", [(3_800, 200), (5_000, 330), (9_000, 260), (16_000, 200), (40_001, 190), (40_000, 36)])
@pytest.mark.parametrize("paired", [False, True])
def test_groups_of_several_fragments_equal_the_oracle(n, hi, paired):
    """Calls large enough that a warp takes 1, 2, 4 and 8 fragments."""
    db, genome, o = database(False, False)
    lens = np.random.default_rng(n).integers(0, hi + 1, n * (2 if paired else 1))
    bases, q, off = batch(genome, [int(x) for x in lens], n)
    check(db, o, bases, q, off, n, dict(confidence=0.1, min_hit_groups=2, paired=paired))


@pytest.mark.parametrize("piece_len", [256, 512, 8192])
@pytest.mark.parametrize("params", [dict(confidence=0.0, min_hit_groups=0),
                                    dict(confidence=0.2, min_hit_groups=2, min_quality=15)],
                         ids=["plain", "quality"])
def test_long_reads_in_pieces_equal_the_oracle(params, piece_len):
    """Reads built to stress the cuts (test_gpu_split.py), and the -K counters
    of their events against those of whole fragments."""
    from kraken_io import GOLDEN, golden_db
    from test_gpu_counters import classify_with_events
    from test_gpu_split import long_reads, use_piece
    db = k2g.Database.open(os.path.join(GOLDEN, "db_a"))
    use_piece(db, piece_len)
    b = long_reads(31, n=50, quals="min_quality" in params, piece=4 * piece_len if piece_len < 2048 else 8192)
    g = golden_db("db_a")
    o = oracle.Oracle(g.hash.cells, g.hash.capacity, g.hash.key_bits, g.hash.value_bits, g.taxo.parent,
                      oracle.index_opts(g.opts.k, g.opts.l, g.opts.spaced_seed_mask, g.opts.toggle_mask))
    r = classify_batch(db, b, params, mode=k2g.MODE_PIPELINED)
    assert r.status == 0
    calls, hg, nr, runs, base = o.classify(b.bases, b.quals, b.seq_off, b.n_frags, threads=4, **params)
    assert np.array_equal(r.call[:b.n_frags], calls.astype(np.uint32))
    assert np.array_equal(r.hit_groups[:b.n_frags], hg.astype(np.uint32))
    for i in range(b.n_frags):
        want = [(int(x["code"]), int(x["count"])) for x in runs[int(base[i]):int(base[i]) + int(nr[i])]]
        assert r.runs_of(i) == want, i
    b.blocks = (np.arange(b.n_frags) // 7).astype(np.uint32)
    outs = []
    for mode in (k2g.MODE_PIPELINED, k2g.MODE_PLAIN):
        c = k2g.Counters(db)
        reads, res, tr, keep = classify_with_events(db, b, dict(quick=False, paired=False, min_quality=0, **{
            k: v for k, v in params.items() if k != "min_quality"}), mode)
        c.add(reads, res)
        outs.append(c.finish())
        c.close()
        del keep
    for x, y in zip(*outs):
        assert np.array_equal(x, y)
    db.close()


@pytest.mark.parametrize("capacity", [5, 8, 13, 61])
def test_tiny_and_full_tables_equal_the_oracle(capacity):
    """Walks that cross the partial last sector, wrap around, or meet every
    cell of a full table."""
    t = torch()
    rng = np.random.default_rng(capacity)
    parent = np.array([0, 0, 1, 1, 2], np.uint64)
    db = k2g.Database.create(k2g.IndexOptions(K, L, MASK, TOGGLE, 1, 1, 0), capacity, 29, 3, parent)
    genome = ACGT[rng.integers(0, 4, 2000)]
    d_seq = to_dev(np.concatenate([genome, np.zeros(16, np.uint8)]))
    off = to_dev(np.array([0, len(genome)], np.uint64))
    mins = t.zeros(len(genome), dtype=t.int64, device="cuda")
    amb = t.zeros(len(genome), dtype=t.uint8, device="cuda")
    st = t.cuda.current_stream().cuda_stream
    db.scan(d_seq.data_ptr(), off.data_ptr(), 1, mins.data_ptr(), amb.data_ptr(), st)
    keys = t.unique(mins[:1966])[:capacity]
    taxa = to_dev(rng.integers(1, 5, capacity).astype(np.uint32))
    db.build_insert(keys.data_ptr(), taxa.data_ptr(), capacity, False, st)
    cells, size = db.download()
    assert size == capacity
    o = oracle.Oracle(cells, capacity, 29, 3, parent, oracle.index_opts(K, L, MASK, TOGGLE))
    bases, q, off = batch(genome, [150] * 60 + [301, 1000], capacity)
    check(db, o, bases, q, off, 62, dict(confidence=0.0, min_hit_groups=1))
    db.close()
