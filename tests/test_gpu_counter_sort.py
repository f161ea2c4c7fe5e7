"""The counters' sorted, distinct entries (export) of any imported ones: bucket
counts and sizes at their edges, and skewed entries that leave the buckets."""
import numpy as np
import pytest

import kraken2_gb300 as k2g

pytestmark = pytest.mark.gpu


def spread(rng, n, nodes, tbits):
    return rng.integers(0, 2**32, n, dtype=np.uint64) << np.uint64(tbits) | rng.integers(1, nodes, n, dtype=np.uint64)


def clumped(rng, n, nodes, tbits, repeats, range_bits):
    """Half spread; half within 2^range_bits encodings, each entry `repeats` times."""
    few = rng.integers(0, 2**range_bits, max(n // 2 // repeats, 1), dtype=np.uint64) << np.uint64(tbits)
    few |= rng.integers(1, nodes, len(few), dtype=np.uint64)
    few += np.uint64(0x9000_0000 << tbits)
    return rng.permutation(np.concatenate([np.repeat(few, repeats), spread(rng, n // 2, nodes, tbits)]))


@pytest.mark.parametrize("nodes", [2, 1000, 70_000])
@pytest.mark.parametrize("n,repeats,range_bits", [
    (0, 0, 0), (1, 0, 0), (2, 0, 0), (4500, 0, 0), (4501, 0, 0), (9002, 0, 0), (1_000_000, 0, 0),
    (40_000, 20_000, 10),     # one entry many times: a zone of 20,000
    (40_000, 1, 12),          # a bucket of 20,000 distinct entries
    (14_000, 1, 14),          # 7,000: one zone of many
    (70_000, 5, 9), (80_000, 40_000, 1),   # a bucket above its limit: the radix sort
    (3_000_000, 3, 20)])
def test_export_is_sorted_and_distinct(n, repeats, range_bits, nodes):
    rng = np.random.default_rng(n + nodes)
    parent = np.concatenate([[0], np.arange(nodes - 1) // 2]).astype(np.uint64)
    db = k2g.Database.create(k2g.IndexOptions(35, 31, 0, 0, 1, 1, 0), 64, 8, 24, parent)
    c = k2g.Counters(db)
    tbits = nodes.bit_length()
    keys = (clumped(rng, n, nodes, tbits, repeats, range_bits) if repeats else spread(rng, n, nodes, tbits)).astype(np.uint64)
    state = {"entries": keys, "taxon_kmers": np.zeros(nodes, np.uint64), "dense": np.zeros(nodes, np.uint8)}
    half = dict(state, entries=keys[: n // 3])
    c.import_state(half)
    assert np.array_equal(c.export()["entries"], np.unique(keys[: n // 3]))
    c.import_state(state)          # on top of the sorted ones
    assert np.array_equal(c.export()["entries"], np.unique(keys))
    assert np.array_equal(c.export()["entries"], np.unique(keys))
    c.close()
    db.close()
