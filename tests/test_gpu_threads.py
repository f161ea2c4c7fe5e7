"""Builds and counters of several threads at a time, which share kernels, the
scratch pool and nothing else: each gives what it gives alone."""
import threading

import numpy as np
import pytest

import kraken2_gb300 as k2g
from gpu_util import torch

pytestmark = pytest.mark.gpu

OPTS = k2g.IndexOptions(35, 31, 0, 0xe37e28c4271b5a2d, 1, 1, 0)
PARENT = np.array([0, 0, 1, 1, 2], np.uint64)


def builder(seed):
    rng = np.random.default_rng(seed)
    seq = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 300_000)]
    off = np.array([0, 100_000, 200_000, 300_000], np.uint64)

    def step():
        db = k2g.Database.create(OPTS, 250_007, 22, 10, PARENT)
        db.build_sequences(seq, off, np.array([2, 3, 4], np.uint32))
        cells, size = db.download()
        counts, _ = db.value_counts()
        db.close()
        return cells, np.array([size]), counts
    return step


def counter(seed):
    rng = np.random.default_rng(seed)
    nodes, n = 400 * seed, 200_000 * seed
    parent = np.concatenate([[0], np.arange(nodes - 1) // 2]).astype(np.uint64)
    db = k2g.Database.create(k2g.IndexOptions(35, 31, 0, 0, 1, 1, 0), 64, 8, 24, parent)
    bits = nodes.bit_length()
    ent = rng.integers(0, 2**32, n, dtype=np.uint64) << np.uint64(bits) | rng.integers(1, nodes, n).astype(np.uint64)
    st = torch().cuda.Stream()

    def step():
        c = k2g.Counters(db)
        c.import_state({"entries": ent, "taxon_kmers": np.ones(nodes, np.uint64), "dense": np.zeros(nodes, np.uint8)},
                       st.cuda_stream)
        out = (c.export(st.cuda_stream)["entries"], *c.finish(st.cuda_stream))
        c.close()
        return out
    return step


def test_threads_do_not_disturb_each_other():
    steps = [builder(1), builder(2), builder(3), counter(1), counter(3)]
    want = [s() for s in steps]
    failed = []

    def run(i):
        try:
            for _ in range(120):
                if not all(np.array_equal(a, b) for a, b in zip(steps[i](), want[i])):
                    failed.append((i, "differs"))
                    return
        except Exception as e:
            failed.append((i, repr(e)))

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(steps))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert failed == []
