"""k2g_classify_host where every one of its slots is used again while others
are under way: long fragments (four slots) and hit events (three), more chunks
than slots, against the same reads in parts of one chunk each."""
import numpy as np
import pytest

import kraken2_gb300 as k2g
from test_gpu_host_chunks import MB, host, make

pytestmark = pytest.mark.gpu


def chunks(off, per, blocks=None):
    """The chunks that the call is cut into (its plan, restated)."""
    n = (len(off) - 1) // per
    total = int(off[-1])
    long_ = total > 512 * n
    most = min(64 * MB if blocks is not None else 128 * MB,
               max((20 if long_ else 16) * MB, total // (4 if blocks is not None else 12) + 1))
    starts = off[::per].astype(np.int64)
    out, f = 0, 0
    while f < n:
        g = max(int(np.searchsorted(starts, starts[f] + most, side="right")) - 1, f + 1)
        if blocks is not None and g < n:
            first = int(np.searchsorted(blocks, blocks[g], side="left"))
            g = first if first > f else int(np.searchsorted(blocks, blocks[g], side="right"))
        out, f = out + 1, g
    return out


@pytest.mark.parametrize("paired", [False, True])
def test_long_fragments_use_every_slot_again(paired):
    per, length = (2 if paired else 1), 5000
    n = 260 * MB // (length * per)
    lens = np.full(n * per, length)
    lens[::7] = 31
    lens[3::11] = 0
    db, off, bases = make(lens, 5)
    assert chunks(off, per) >= 9                       # four slots, each at least twice
    s, call, hg, hlen, runs, tr = host(db, off, bases, 0, n, paired)
    k2g.check(s)
    step = 9 * MB // (length * per)
    parts = [host(db, off, bases, f, min(f + step, n), paired) for f in range(0, n, step)]
    for p in parts:
        k2g.check(p[0])
    for i, whole in ((1, call), (2, hg), (3, hlen), (4, runs)):
        assert np.array_equal(whole, np.concatenate([p[i] for p in parts]))
    assert np.array_equal(tr, sum(p[5] for p in parts)) and (call > 0).any()
    again = host(db, off, bases, 0, n, paired, runs_cap=len(runs))
    k2g.check(again[0])
    assert np.array_equal(again[4], runs) and np.array_equal(again[1], call)
    db.close()


@pytest.mark.parametrize("length", [150, 5000])
def test_hit_events_use_every_slot_again(length):
    n = 450 * MB // length
    off = np.arange(n + 1, dtype=np.uint64) * np.uint64(length)
    db, off, bases = make(np.full(n, length), 6)
    block = 3 * MB // length
    blocks = (np.arange(n) // block).astype(np.uint32)
    assert chunks(off, 1, blocks) >= 7                 # three slots, each at least twice
    whole = k2g.Counters(db)
    s, call, hg, hlen, runs, tr = host(db, off, bases, 0, n, False, blocks, whole)
    k2g.check(s)
    parts = k2g.Counters(db)
    step = 2 * block
    got = []
    for f in range(0, n, step):
        p = host(db, off, bases, f, min(f + step, n), False, blocks, parts)
        k2g.check(p[0])
        got.append(p)
    for i, w in ((1, call), (2, hg), (3, hlen), (4, runs)):
        assert np.array_equal(w, np.concatenate([p[i] for p in got]))
    assert np.array_equal(tr, sum(p[5] for p in got))
    assert all(np.array_equal(a, b) for a, b in zip(whole.finish(), parts.finish()))
    db.close()
