"""Fragments with more taxa than a warp's maps in shared memory hold, which are
resolved from a map in the unused part of their run region: against the oracle,
and in a time that does not grow with the square of their runs."""
import time

import numpy as np
import pytest

import kraken2_gb300 as k2g
import test_gpu_warp as warp
import test_gpu_warp_translated as translated
from gpu_util import bytes_dev, to_dev, torch, zeros

pytestmark = pytest.mark.gpu


# 512 taxa fit the largest map in shared memory: about 1,550 bases of one taxon
# a k-mer; then maps of 1,024 slots and more
@pytest.mark.parametrize("length,n", [(1400, 40), (1500, 40), (1600, 40), (1700, 40), (3100, 30), (4095, 30)])
@pytest.mark.parametrize("confidence", [0.0, 0.3])
def test_single_fragments(length, n, confidence):
    db, genome, o = warp.database(False, True)
    bases, q, off = warp.batch(genome, [length - i % 3 for i in range(n)], length)
    warp.check(db, o, bases, q, off, n, dict(confidence=confidence, min_hit_groups=2))


@pytest.mark.parametrize("length,n", [(800, 40), (2000, 20), (9001, 10)])
def test_pairs(length, n):
    db, genome, o = warp.database(False, True)
    bases, q, off = warp.batch(genome, [length + i % 5 for i in range(2 * n)], length)
    warp.check(db, o, bases, q, off, n, dict(confidence=0.05, min_hit_groups=2, paired=True))


@pytest.mark.parametrize("paired", [False, True])
def test_translated(paired):
    db, genome, o = translated.database(False, True)
    lens = [20_000, 27_000, 30_001, 41_000, 60_002, 79_999] * 2
    bases, q, off = warp.batch(genome, lens, 4)
    warp.check(db, o, bases, q, off, len(lens) // (2 if paired else 1),
               dict(confidence=0.02, min_hit_groups=2, paired=paired))


def test_pairs_of_long_reads_take_no_quadratic_time():
    """Against the fused kernel, which counts into a map as well (and was 3.8
    times as fast as the runs compared with each other)."""
    t = torch()
    db, genome, _ = warp.database(False, True)
    n, length = 200, 50_000
    bases, _, off = warp.batch(genome, [length] * (2 * n), 1)
    d_b, d_o = bytes_dev(bases), to_dev(off)
    cap = int(off[-1]) + 2 * n + 8
    out = [zeros(n, t.int32), zeros(cap, t.int64), zeros(1, t.int32)]
    reads = k2g.Reads(d_b.data_ptr(), None, d_o.data_ptr(), n, length, int(off[-1]), None, 0)
    res = k2g.Results(out[0].data_ptr(), None, None, None, out[1].data_ptr(), cap, None, None, None, None, 0, None,
                      out[2].data_ptr())
    best, calls = {}, {}
    for mode in (k2g.MODE_PERSISTENT, k2g.MODE_PIPELINED):
        for _ in range(3):
            t.cuda.synchronize()
            t0 = time.perf_counter()
            db.classify(reads, k2g.ClassifyParams(0.1, 2, 0, 1, 0), res, mode=mode,
                        stream=t.cuda.current_stream().cuda_stream)
            t.cuda.synchronize()
            best[mode] = min(best.get(mode, 1e9), time.perf_counter() - t0)
        calls[mode] = out[0].cpu().numpy()
    assert np.array_equal(calls[k2g.MODE_PERSISTENT], calls[k2g.MODE_PIPELINED]) and int(out[2][0]) == 0
    assert best[k2g.MODE_PIPELINED] < 2 * best[k2g.MODE_PERSISTENT]
