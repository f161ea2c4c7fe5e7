"""Settings that all threads of a process share (on the fake runtime): a call
leaves none lower than it found it, so that calls of several threads may set
and launch in any order."""
import ctypes as C

import numpy as np

import kraken2_gb300 as k2g
from fake_cuda import fake_cuda

OPTS = k2g.IndexOptions(35, 31, 0, 0xe37e28c4271b5a2d, 1, 1, 0)
PARENT = np.array([0, 0, 1, 1, 2], np.uint64)


def test_limits_of_shared_memory_are_not_lowered():
    with fake_cuda() as f:
        db = k2g.Database.create(OPTS, 100_003, 22, 10, PARENT, device=60)
        large = k2g.Database.create(OPTS, 100_003, 16, 16, np.arange(50_000, dtype=np.uint64) // 2, device=60)

        def found(name, args):       # enough candidates, and one large bucket
            if "block_scan_kernel" in name:
                last = C.cast(args[3], C.POINTER(C.c_uint64))[0] - 1
                C.cast(C.cast(args[5], C.POINTER(C.c_void_p))[0], C.POINTER(C.c_uint32))[last] = 20_000
            if "bucket_largest_kernel" in name:
                C.cast(C.cast(args[2], C.POINTER(C.c_void_p))[0], C.POINTER(C.c_uint32))[0] = 20_000

        f.hook(found)
        seq, off = np.zeros(40_000, np.uint8), np.array([0, 40_000], np.uint64)
        state = {"entries": np.arange(1, 20_001, dtype=np.uint64) << np.uint64(3), "taxon_kmers": np.zeros(5, np.uint64),
                 "dense": np.zeros(5, np.uint8)}
        st = f.stream()
        for _ in range(2):
            db.build_sequences(seq, off, np.array([3], np.uint32))
            c = k2g.Counters(db)
            c.import_state(state, st)
            c.export(st)
            c.close()
            large.value_counts(st)
            db.value_counts(st)
        assert f.launches("bucket_sort_kernel") == 8 and f.launches("value_hist_kernel") >= 4
        db.close()
        large.close()
        assert f.faults() == []
