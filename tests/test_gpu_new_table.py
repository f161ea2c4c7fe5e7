"""A small library put into a table of several GB straight after its creation,
which has to wait until the device has cleared the cells: the same table as one
built after a synchronisation of the whole device."""
import numpy as np
import pytest

import kraken2_gb300 as k2g
from gpu_util import to_dev, torch, u32, zeros

pytestmark = pytest.mark.gpu

CAPACITY = 1_500_000_007                  # 6 GB: about a millisecond to clear
ACGT = np.frombuffer(b"ACGT", np.uint8)
PARENT = np.array([0, 0, 1, 1, 2, 2], np.uint64)


def build(seq, wait, how, mins):
    t = torch()
    db = k2g.Database.create(k2g.IndexOptions(35, 31, 0, 0xe37e28c4271b5a2d, 1, 1, 0), CAPACITY, 22, 10, PARENT)
    if wait:
        t.cuda.synchronize()
    if how == "insert":                   # a caller's own stream
        st = t.cuda.Stream()
        db.build_insert(mins[0].data_ptr(), mins[1].data_ptr(), len(mins[0]), False, st.cuda_stream)
        t.cuda.synchronize()
    else:
        off = np.array([0, len(seq) // 2, len(seq)], np.uint64)
        db.build_sequences(seq, off, np.array([4, 5], np.uint32), ordered=how == "ordered")
    return db


@pytest.mark.parametrize("how", ["ordered", "unordered", "insert"])
def test_build_right_after_creation(how):
    t = torch()
    rng = np.random.default_rng(3)
    seq = ACGT[rng.integers(0, 4, 60_000)]
    probe = k2g.Database.create(k2g.IndexOptions(35, 31, 0, 0xe37e28c4271b5a2d, 1, 1, 0), 1009, 22, 10, PARENT)
    mins, amb = zeros(len(seq) + 1, t.int64), zeros(len(seq) + 1, t.uint8)
    d_b, d_o = to_dev(np.concatenate([seq, np.zeros(16, np.uint8)])), to_dev(np.array([0, len(seq)], np.uint64))
    probe.scan(d_b.data_ptr(), d_o.data_ptr(), 1, mins.data_ptr(), amb.data_ptr(),
               t.cuda.current_stream().cuda_stream)
    n = len(seq) - 34
    pairs = (mins[:n].contiguous(), to_dev((np.arange(n) % 5 + 1).astype(np.uint32)))
    t.cuda.synchronize()
    got = []
    for wait in (False, True):
        db = build(seq, wait, how, pairs)
        vals = zeros(n, t.int32)
        db.lookup(pairs[0].data_ptr(), vals.data_ptr(), n, t.cuda.current_stream().cuda_stream)
        t.cuda.synchronize()
        got.append((u32(vals).copy(), int(db.info().size)))
        db.close()
    assert np.array_equal(got[0][0], got[1][0]) and got[0][1] == got[1][1] > n // 4
    if how == "insert":
        assert (got[0][0] > 0).all()
