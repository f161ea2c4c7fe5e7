"""Which sort k2g_build_sequences takes (on the fake runtime): blocks of few
candidates, short sequences, go to the radix passes, which do not mind how
many blocks there are."""
import ctypes as C

import numpy as np
import pytest

import kraken2_gb300 as k2g
from fake_cuda import fake_cuda

PARENT = np.array([0, 0, 1, 1, 2], np.uint64)


@pytest.mark.parametrize("per_block,by_blocks", [(1, False), (23, False), (24, True), (500, True)])
def test_sort_by_candidates_a_block(per_block, by_blocks):
    with fake_cuda() as f:
        db = k2g.Database.create(k2g.IndexOptions(35, 31, 0, 0, 1, 1, 0), 100_003, 22, 10, PARENT, device=58)
        n = 100

        def found(name, args):       # the scan's counts, one chunk a sequence
            if "block_scan_kernel" in name:
                counts = C.cast(C.cast(args[5], C.POINTER(C.c_void_p))[0], C.POINTER(C.c_uint32))
                # (the exclusive scan does nothing here: the last count is added to itself)
                counts[n - 1] = per_block * n // 2

        f.hook(found)
        off = np.arange(n + 1, dtype=np.uint64) * np.uint64(1000)
        db.build_sequences(np.zeros(n * 1000, np.uint8), off, np.full(n, 3, np.uint32), subblock_size=16384)
        assert (f.launches("bucket_sort_kernel") > 0) == by_blocks
        assert (f.launches("pair_scatter_kernel") > 0) == (not by_blocks)
        db.close()
