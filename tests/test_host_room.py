"""Bases are read as the 16-byte chunks that contain them: the library's own
buffers have to reach to the end of the last one (on the fake runtime)."""
import ctypes as C

import numpy as np
import pytest

import kraken2_gb300 as k2g
from fake_cuda import fake_cuda

OPTS = k2g.IndexOptions(35, 31, 0, 0xe37e28c4271b5a2d, 1, 1, 0)
PARENT = np.array([0, 0, 1, 1, 2], np.uint64)


@pytest.mark.parametrize("total", [100_000, 100_001, 100_007, 100_009, 100_015])
@pytest.mark.parametrize("what", ["sequences", "sample", "host"])
def test_the_last_chunk_lies_inside_the_buffer(what, total):
    with fake_cuda() as f:
        db = k2g.Database.create(OPTS, 100_003, 22, 10, PARENT, device=55)
        seq, off = np.full(total, ord("A"), np.uint8), np.array([0, total], np.uint64)
        if what == "sequences":
            db.build_sequences(seq, off, np.array([3], np.uint32))
        elif what == "sample":
            db.sample_minimizers(seq, off)
        else:
            call, cp = np.zeros(1, np.uint32), k2g.ClassifyParams(0.0, 2, 0, 0, 0)
            k2g.check(k2g.lib().k2g_classify_host(db.h, seq.ctypes.data, None, off.ctypes.data, 1, C.byref(cp),
                                                  call.ctypes.data, None, None, None, None, None))
        assert f.tail_of_copy(total) >= -total % 16
        db.close()
