"""Tables whose taxonomy has several roots: the staged kernels with the default
window (words of four bases, with and without a least hash and qualities)
against the oracle, and fragments whose best taxa lie in different trees."""
import os

import numpy as np
import pytest

import kraken2_gb300 as k2g
import oracle
import test_gpu_warp as warp
from gpu_util import classify_batch, to_dev, torch
from kraken_io import Batch

pytestmark = pytest.mark.gpu

K, L, MASK, TOGGLE, ACGT = warp.K, warp.L, warp.MASK, warp.TOGGLE, warp.ACGT
_cache = {}


def table(parent, genome, taxa, min_hash=0, wide=False):
    """A table of the genome's minimizers, k-mer i's with taxa[i]."""
    t = torch()
    vb = 12
    db = k2g.Database.create(k2g.IndexOptions(K, L, MASK, TOGGLE, 1, 1, min_hash), 200_003, (40 if wide else 32) - vb,
                             vb, parent)
    st = t.cuda.current_stream().cuda_stream
    d_seq = to_dev(np.concatenate([genome, np.zeros(16, np.uint8)]))
    mins = t.zeros(len(genome), dtype=t.int64, device="cuda")
    amb = t.zeros(len(genome), dtype=t.uint8, device="cuda")
    d_off = to_dev(np.array([0, len(genome)], np.uint64))
    db.scan(d_seq.data_ptr(), d_off.data_ptr(), 1, mins.data_ptr(), amb.data_ptr(), st)
    d_tax = to_dev(taxa.astype(np.uint32))
    db.build_insert(mins.data_ptr(), d_tax.data_ptr(), len(taxa), True, st)
    t.cuda.synchronize()
    return db


def staged_table(min_hash, wide):
    """As test_gpu_warp's, with a last node that is a root of its own and has
    no k-mers: no result depends on the order in which taxa are joined."""
    if (min_hash, wide) not in _cache:
        rng = np.random.default_rng(17)
        genome = ACGT[rng.integers(0, 4, 120_000)]
        nodes = 4000
        parent = np.zeros(nodes, np.uint64)
        parent[2:-1] = (rng.random(nodes - 3) * np.minimum(np.arange(1, nodes - 2), 300)).astype(np.uint64) + 1
        n = len(genome) - K + 1
        taxa = np.repeat(rng.integers(1, nodes - 1, n), rng.integers(60, 2000, n))[:n]
        taxa[rng.random(n) < 0.3] = 0
        db = table(parent, genome, taxa, min_hash, wide)
        cells, _ = db.download()
        inf = db.info()
        o = oracle.Oracle(cells, inf.capacity, inf.key_bits, inf.value_bits, parent,
                          oracle.index_opts(K, L, MASK, TOGGLE, 1, min_hash))
        _cache[min_hash, wide] = db, genome, o
    return _cache[min_hash, wide]


def check(db, o, bases, q, off, n, params):
    b = Batch(bases, q, off, n, params.get("paired", False), [""] * n, [(0,)] * n, np.zeros(n, np.uint32))
    r = classify_batch(db, b, params)
    assert r.status == 0
    calls, hg, nr, runs, base = o.classify(bases, q, off, n, threads=os.cpu_count() or 1, **params)
    assert np.array_equal(r.call[:n], calls.astype(np.uint32))
    assert np.array_equal(r.hit_groups[:n], hg.astype(np.uint32))
    nr = nr.astype(np.int64)
    assert np.array_equal(r.hitlist_len[:n], nr)
    within = np.arange(int(nr.sum())) - np.repeat(np.cumsum(nr) - nr, nr)
    got = r.runs[np.repeat(r.hitlist_off[:n].astype(np.int64), nr) + within]
    want = runs[np.repeat(base.astype(np.int64), nr) + within]
    assert np.array_equal(got >> np.uint64(32), want["code"].astype(np.uint64) & np.uint64(0xFFFFFFFF))
    assert np.array_equal(got & np.uint64(0xFFFFFFFF), want["count"].astype(np.uint64))


@pytest.mark.parametrize("min_hash", [0, 1 << 62])
@pytest.mark.parametrize("params", warp.PARAMS, ids=lambda p: "-".join(f"{k}{v}" for k, v in p.items()))
def test_staged_kernels_match_the_oracle(params, min_hash):
    db, genome, o = staged_table(min_hash, False)
    rng = np.random.default_rng(len(params) + (min_hash > 0))
    per = 2 if params.get("paired") else 1
    for lens in (np.array(warp.EDGES), np.full(2000, 150), rng.integers(20, 301, 3001), rng.integers(30, 3000, 400)):
        lens = np.resize(lens, len(lens) + len(lens) % per)
        bases, q, off = warp.batch(genome, [int(x) for x in lens], 3, quals="min_quality" in params)
        check(db, o, bases, q, off, len(lens) // per, params)


@pytest.mark.parametrize("trees", [2, 3])
@pytest.mark.parametrize("mode", [k2g.MODE_PLAIN, k2g.MODE_PERSISTENT, k2g.MODE_PIPELINED])
def test_best_taxa_in_different_trees(mode, trees):
    """Joined one after another: two give 0, a third gives itself."""
    rng = np.random.default_rng(9)
    genome = ACGT[rng.integers(0, 4, 3000)]
    taxa = np.repeat([4, 5, 6], 1000)[:len(genome) - K + 1]
    taxa[np.arange(len(taxa)) % 1000 > 900] = 0   # (no minimizer of two trees, whose LCA would be 0)
    db = table(np.array([0, 0, 0, 0, 1, 2, 3], np.uint64), genome, taxa)
    # as many k-mers of each tree's taxon (behind an ambiguous base the reference counts one early)
    part = [bytes(genome[i * 1000 + 200:i * 1000 + (321 if i == 0 else 320)]) for i in range(trees)]
    read = b"N".join(part)
    n = 40
    off = np.arange(n + 1, dtype=np.uint64) * np.uint64(len(read))
    b = Batch(read * n, None, off, n, False, [""] * n, [(0,)] * n, np.zeros(n, np.uint32))
    r = classify_batch(db, b, dict(confidence=0.0, min_hit_groups=1), mode=mode)
    assert r.status == 0 and (r.hit_groups[:n] > 0).all()
    assert {m for code, m in r.runs_of(0) if code in (4, 5, 6)} == {87}
    calls = set(r.call[:n].tolist())
    assert calls == {0} if trees == 2 else calls <= {4, 5, 6}
    db.close()
