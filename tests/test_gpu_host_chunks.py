"""k2g_classify_host and _blocks over several chunks: results, runs, per-taxon
counts and counters equal those of one chunk per call (the same reads in
parts), a runs buffer that is too small is refused, and the next call works."""
import ctypes as C

import numpy as np
import pytest

import kraken2_gb300 as k2g
from gpu_util import to_dev, torch

pytestmark = pytest.mark.gpu

MB = 1 << 20
NODES = 400


def make(lens, seed):
    rng = np.random.default_rng(seed)
    parent = np.concatenate([[0], np.arange(NODES - 1) // 2]).astype(np.uint64)
    db = k2g.Database.create(k2g.IndexOptions(35, 31, 0, 0xe37e28c4271b5a2d, 1, 1, 0), 1_000_003, 22, 10, parent)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    bases = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, int(off[-1]) + 16, dtype=np.uint8)]
    t = torch()
    mins, amb = t.zeros(4_000_000, dtype=t.int64, device="cuda"), t.zeros(4_000_000, dtype=t.uint8, device="cuda")
    st = t.cuda.current_stream().cuda_stream
    d_b, d_o = to_dev(bases[:4_000_016]), to_dev(np.array([0, 4_000_000], np.uint64))
    db.scan(d_b.data_ptr(), d_o.data_ptr(), 1, mins.data_ptr(), amb.data_ptr(), st)
    keys = np.unique(mins.cpu().numpy()[:3_999_900:4])[:600_000]
    d_k, d_t = to_dev(keys.view(np.uint64)), to_dev(rng.integers(1, NODES, len(keys)).astype(np.uint32))
    db.build_insert(d_k.data_ptr(), d_t.data_ptr(), len(keys), False, st)
    t.cuda.synchronize()
    # every chunk meets stored k-mers
    bases = np.resize(bases[:4_000_000], int(off[-1]) + 16)
    return db, off, bases


def host(db, off, bases, f0, f1, paired, blocks=None, counters=None, runs_cap=None):
    per = 2 if paired else 1
    n = f1 - f0
    part = np.ascontiguousarray(off[f0 * per:f1 * per + 1])
    call, hg, hlen = (np.zeros(max(n, 1), np.uint32) for _ in range(3))
    runs = np.zeros(int(part[-1] - part[0]) + 2 * n + 8 if runs_cap is None else runs_cap, np.uint64)
    nr = C.c_uint64(len(runs))
    tr = np.zeros(NODES, np.uint64)
    cp = k2g.ClassifyParams(0.05, 2, 0, int(paired), 0)
    out = (C.byref(cp), call.ctypes.data, hg.ctypes.data, hlen.ctypes.data, runs.ctypes.data, C.byref(nr),
           tr.ctypes.data)
    if counters is None:
        s = k2g.lib().k2g_classify_host(db.h, bases.ctypes.data, None, part.ctypes.data, n, *out)
    else:
        s = k2g.lib().k2g_classify_host_blocks(db.h, bases.ctypes.data, None, part.ctypes.data, n,
                                               blocks[f0:f1].ctypes.data, counters.h, *out)
    return s, call, hg, hlen, runs[:nr.value].copy(), tr


@pytest.mark.parametrize("total_mb", [3, 20, 36, 52, 100])          # 1, 2, 3, 4 and 7 chunks
@pytest.mark.parametrize("paired", [False, True])
@pytest.mark.parametrize("length", [150, 5000])                       # short and long lists of runs
def test_chunks_equal_parts(total_mb, paired, length):
    per = 2 if paired else 1
    n = total_mb * MB // (length * per)
    lens = np.full(n * per, length)
    lens[::7] = 31
    lens[3::11] = 0
    db, off, bases = make(lens, total_mb)
    s, call, hg, hlen, runs, tr = host(db, off, bases, 0, n, paired)
    k2g.check(s)
    step = 9 * MB // (length * per)                                    # parts of one chunk each
    parts = [host(db, off, bases, f, min(f + step, n), paired) for f in range(0, n, step)]
    for p in parts:
        k2g.check(p[0])
    for i, whole in ((1, call), (2, hg), (3, hlen), (4, runs)):
        assert np.array_equal(whole, np.concatenate([p[i] for p in parts]))
    assert np.array_equal(tr, sum(p[5] for p in parts))
    assert (call > 0).any() and len(runs) == int(hlen.sum(dtype=np.int64))

    s, *_ = host(db, off, bases, 0, n, paired, runs_cap=len(runs) - 1)
    assert s != 0
    again = host(db, off, bases, 0, n, paired, runs_cap=len(runs))
    k2g.check(again[0])
    assert np.array_equal(again[4], runs) and np.array_equal(again[1], call)
    db.close()


@pytest.mark.parametrize("total_mb,block_frags", [(3, 700), (40, 997), (90, 20_000), (40, 10**9)])
def test_counters_over_chunks_equal_parts(total_mb, block_frags):
    n = total_mb * MB // 150
    db, off, bases = make(np.full(n, 150), total_mb)
    blocks = (np.arange(n) // block_frags).astype(np.uint32)
    whole = k2g.Counters(db)
    s, call, *_ = host(db, off, bases, 0, n, False, blocks, whole)
    k2g.check(s)
    parts = k2g.Counters(db)
    step = max(8 * MB // 150 // block_frags, 1) * block_frags          # ends at block boundaries
    calls = []
    for f in range(0, n, step):
        p = host(db, off, bases, f, min(f + step, n), False, blocks, parts)
        k2g.check(p[0])
        calls.append(p[1])
    assert np.array_equal(call, np.concatenate(calls))
    assert all(np.array_equal(a, b) for a, b in zip(whole.finish(), parts.finish()))
    db.close()
