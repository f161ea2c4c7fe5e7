"""The counters' sort where a few minimizers make up most events, as in a sample
of one small genome: the distinct entries, in a time near that of as many
events of all different ones."""
import ctypes as C
import time

import numpy as np
import pytest

import kraken2_gb300 as k2g

pytestmark = pytest.mark.gpu
NODES = 2000
TBITS = NODES.bit_length()
PARENT = np.concatenate([[0, 0], np.ones(NODES - 2)]).astype(np.uint64)


def entries(rng, n):
    return rng.integers(0, 2**32, n, dtype=np.uint64) << np.uint64(TBITS) | rng.integers(1, NODES, n).astype(np.uint64)


def export_time(db, ent):
    """(seconds of the sort, the entries left)"""
    c = k2g.Counters(db)
    c.import_state({"entries": ent, "taxon_kmers": np.zeros(NODES, np.uint64), "dense": np.zeros(NODES, np.uint8)})
    m = C.c_uint64()
    t0 = time.perf_counter()
    k2g.check(k2g.lib().k2g_counters_export(c.h, None, 0, C.byref(m), None, None, None))
    t0 = time.perf_counter() - t0
    got = c.export()["entries"]
    c.close()
    return t0, got


@pytest.fixture(scope="module")
def db():
    d = k2g.Database.create(k2g.IndexOptions(35, 31, 0, 0, 1, 1, 0), 64, 8, 24, PARENT)
    yield d
    d.close()


# a zone's keys: of 1, 2, 16 to 40 distinct ones, even and uneven; more than
# are taken out one by one; with and without others left over
@pytest.mark.parametrize("distinct", [1, 2, 16, 31, 32, 33, 40, 1000, 30_000])
@pytest.mark.parametrize("n", [33, 3000, 20_000, 300_000])
@pytest.mark.parametrize("uneven", [False, True])
def test_few_distinct_entries(db, distinct, n, uneven):
    rng = np.random.default_rng(distinct + n)
    keys = entries(rng, distinct)
    if distinct <= 40:      # in one zone: the same upper bits
        keys = (keys & np.uint64((1 << (TBITS + 4)) - 1)) | np.uint64(0x8123_4560 << TBITS)
        keys = np.where((keys & np.uint64((1 << TBITS) - 1)) == 0, keys + np.uint64(1), keys)
        keys = (keys >> np.uint64(TBITS) << np.uint64(TBITS)) | (keys & np.uint64((1 << TBITS) - 1)) % np.uint64(NODES)
    share = rng.pareto(1.0, distinct) + 0.01 if uneven else np.ones(distinct)
    ent = keys[rng.choice(distinct, n, p=share / share.sum())]
    _, got = export_time(db, ent)
    assert np.array_equal(got, np.unique(ent))


@pytest.mark.parametrize("n,distinct", [(300_000, 30), (3_000_000, 1000), (28_000_000, 10_000), (28_000_000, 1)])
def test_repeats_cost_little(db, n, distinct):
    """(they took 12, 5, 7 and 13 times as long)"""
    rng = np.random.default_rng(n)
    keys = entries(rng, distinct)
    few, all_ = keys[rng.integers(0, distinct, n)], entries(rng, n)
    best = [min(export_time(db, x)[0] for _ in range(3)) for x in (few, all_)]
    assert best[0] < 4 * best[1]
