"""k2g_build_sequences at the edges of its blocks and of the shared-memory
sort: block sizes that leave and meet the sort's limits, subblocks, ambiguous
bases, repeats.  The table equals one filled in order with the list made here
from k2g_scan's minimizers: block after block, a block's distinct ones by zone
(MurmurHash3 mod 256) and value."""
import numpy as np
import pytest

import kraken2_gb300 as k2g
from gpu_util import to_dev, torch, zeros
from kraken_io import murmur3_np

pytestmark = pytest.mark.gpu
K, L = 35, 31
TOGGLE = 0xe37e28c4271b5a2d


def new_db(nodes, k=K, capacity=1_000_003, key_bits=20, one_root=True):
    parent = np.arange(nodes, dtype=np.uint64) // 2
    if not one_root:
        parent[2] = 0
    return k2g.Database.create(k2g.IndexOptions(k, L, 0, TOGGLE, 1, 1, 0), capacity, key_bits, 32 - key_bits, parent)


def scan(db, bases, k):
    """(minimizer, ambiguous) of every k-mer of one sequence, by k2g_scan."""
    t = torch()
    n = len(bases)
    mins, amb = zeros(n + 1, t.int64), zeros(n + 1, t.uint8)
    d_b, d_o = to_dev(np.concatenate([bases, np.zeros(16, np.uint8)])), to_dev(np.array([0, n], np.uint64))
    db.scan(d_b.data_ptr(), d_o.data_ptr(), 1, mins.data_ptr(), amb.data_ptr(), t.cuda.current_stream().cuda_stream)
    m = max(n - k + 1, 0)
    return mins.cpu().numpy().view(np.uint64)[:m], amb.cpu().numpy()[:m] != 0


def library(kind, rng):
    acgt = np.frombuffer(b"ACGT", np.uint8)
    if kind == "random":
        lens = [34, 35, 36, 1, 0, 2047, 2048, 2049, 16384 + 34, 16384 + 35, 40_000, 100_003]
    elif kind == "large":
        lens = [150_000, 70_001]
    else:
        lens = [30_000, 20_000, 9_000]
    seqs = [acgt[rng.integers(0, 4, n)] for n in lens]
    if kind == "repeats":
        seqs[0] = np.resize(seqs[0][:61], 30_000)                       # few minimizers, many times
        seqs[1] = np.full(20_000, ord("A"), np.uint8)
        seqs[2] = np.concatenate([seqs[2][:4500], seqs[2][:4500]])
    if kind == "ambiguous":
        for s in seqs:
            s[rng.integers(0, len(s), len(s) // 150)] = ord("N")
            s[1000:1040] = ord("n")
            s[5000:6000] |= 0x20
    return seqs


@pytest.mark.parametrize("kind", ["random", "large", "repeats", "ambiguous"])
@pytest.mark.parametrize("block,sub", [(16384, 1024), (25_600, 25_600), (25_000, 700), (24_576, 1024), (40_000, 1000),
                                       (8064, 8064), (500, 64), (3000, 1)])
def test_list_equals_scan_by_hand(kind, block, sub):
    rng = np.random.default_rng(block + sub)
    seqs = library(kind, rng)
    nodes = len(seqs) + 2
    one_root = block != 25_000   # (several roots: every pair is sorted and replayed)
    db, db1 = new_db(nodes, one_root=one_root), new_db(nodes, k=K - 1)
    off = np.concatenate([[0], np.cumsum([len(s) for s in seqs])]).astype(np.uint64)
    taxa = (np.arange(len(seqs)) + 2).astype(np.uint32)
    taxa[-1] = 1
    n = db.build_sequences(np.concatenate(seqs), off, taxa, block_size=block, subblock_size=sub)
    keys, values = [], []
    for s, tax in zip(seqs, taxa):
        if len(s) < K:
            continue
        mins, amb = scan(db, s, K)
        # a subblock start: the minimizer of the k - l l-mers in its first
        # k - 1 bases, which are all A/C/G/T
        starts, _ = scan(db1, s, K - 1)
        bad = np.concatenate([[0], np.cumsum(~np.isin(s, np.frombuffer(b"ACGTacgt", np.uint8)))])
        good = bad[K - 1:] == bad[:len(bad) - (K - 1)]
        for j in range(0, len(s), block):
            to, end = min(j + block, len(mins)), min(j + block + K - 1, len(s))
            at = np.arange(j, max(end - (K - 1) + 1, j), sub)
            at = at[at >= 1]
            at = at[good[at]]
            found = [mins[j:to][~amb[j:to]], starts[at]]
            u = np.unique(np.concatenate(found))
            zone = (murmur3_np(u) & np.uint64(255)).astype(np.int64)
            keys.append(u[np.lexsort((u, zone))])
            values.append(np.full(len(u), tax, np.uint32))
    keys, values = np.concatenate(keys), np.concatenate(values)
    assert n == len(keys)
    ref = new_db(nodes, one_root=one_root)
    d_k, d_v = to_dev(keys), to_dev(values)
    ref.build_insert(d_k.data_ptr(), d_v.data_ptr(), len(keys), True, torch().cuda.current_stream().cuda_stream)
    a, b = db.download(), ref.download()
    assert np.array_equal(a[0], b[0]) and a[1] == b[1]
    for x in (db, db1, ref):
        x.close()


def test_batches_equal_one_batch():
    """The second batch starts from a table that is not empty."""
    rng = np.random.default_rng(5)
    seqs = library("random", rng)
    seqs += [s.copy() for s in seqs[-2:]]                                # repeated under other taxa
    taxa = (np.arange(len(seqs)) + 2).astype(np.uint32)
    one, two = new_db(len(seqs) + 2), new_db(len(seqs) + 2)

    def add(db, a, b):
        off = np.concatenate([[0], np.cumsum([len(s) for s in seqs[a:b]])]).astype(np.uint64)
        return db.build_sequences(np.concatenate(seqs[a:b]), off, taxa[a:b])

    n = add(one, 0, len(seqs))
    assert add(two, 0, 9) + add(two, 9, 11) + add(two, 11, len(seqs)) == n
    a, b = one.download(), two.download()
    assert np.array_equal(a[0], b[0]) and a[1] == b[1]
    one.close()
    two.close()


@pytest.mark.parametrize("load", [0.05, 0.3, 0.7, 0.95, 1.0])
@pytest.mark.parametrize("key_bits", [6, 22])            # many and few compacted keys that collide
@pytest.mark.parametrize("capacity", [33, 1024, 60_001])
def test_ordered_insert_equals_sequential(load, key_bits, capacity):
    """Clusters with and without moved pairs, across words and the table's
    end, in three batches, against a sequential insert."""
    rng = np.random.default_rng(int(load * 100) + capacity)
    nodes = 60
    db = new_db(nodes, capacity=capacity, key_bits=key_bits)
    distinct = rng.integers(0, 2**62, max(int(capacity * load), 1), dtype=np.int64).astype(np.uint64)
    keys = distinct[rng.integers(0, len(distinct), 3 * len(distinct) + 5)]
    keys[:len(distinct)] = distinct
    taxa = rng.integers(0, nodes, len(keys)).astype(np.uint32)
    parent = np.arange(nodes) // 2
    cells = np.zeros(capacity, np.uint32)
    hc = murmur3_np(keys)
    size = 0
    for h, t in zip(hc.tolist(), taxa.tolist()):
        if not t:
            continue
        at, ck = h % capacity, h >> (64 - key_bits)
        while cells[at] and int(cells[at]) >> (32 - key_bits) != ck:
            at = (at + 1) % capacity
        a, b = int(cells[at]) & ((1 << (32 - key_bits)) - 1), t
        size += not a
        while a and a != b:
            a, b = (int(parent[a]), b) if a > b else (a, int(parent[b]))
        cells[at] = ck << (32 - key_bits) | b
    st = torch().cuda.current_stream().cuda_stream
    cut = [0, len(keys) // 3, 2 * len(keys) // 3, len(keys)]
    if size == capacity:   # a full table is refused by the insert
        cut = cut[:1]
    for x, y in zip(cut, cut[1:]):
        d_k, d_t = to_dev(keys[x:y]), to_dev(taxa[x:y])
        db.build_insert(d_k.data_ptr(), d_t.data_ptr(), y - x, True, st)
    if size < capacity:
        got, n = db.download()
        assert np.array_equal(got, cells) and n == size
    db.close()
