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


@pytest.mark.parametrize("key_bits,load,n,pick", [
    (22, 0.26, 20_000, True), (22, 0.85, 20_000, True), (8, 0.4, 20_000, True), (6, 0.4, 40_000, False),
    (10, 0.66, 20_000, True), (8, 0.66, 20_000, False), (12, 0.85, 20_000, True), (9, 0.85, 20_000, False),
    (10, 0.66, 400_000, False), (22, 1.0, 20_000, True), (6, 1.0, 20_000, False)])
def test_pairs_are_picked_unless_merges_are_expected(key_bits, load, n, pick):
    with fake_cuda() as f:
        capacity = 1_000_003
        db = k2g.Database.create(k2g.IndexOptions(35, 31, 0, 0, 1, 1, 0), capacity, key_bits, 32 - key_bits, PARENT,
                                 device=59)

        def inserted(name, args):    # the size after the unordered pass
            if "13insert_kernel" in name:
                size = C.cast(args[7], C.POINTER(C.c_void_p))[0]
                C.cast(size, C.POINTER(C.c_uint64))[0] = int(load * capacity)

        f.hook(inserted)
        db.build_insert(f.device(np.arange(n, dtype=np.uint64)), f.device(np.ones(n, np.uint32)), n, True, f.stream())
        assert (f.launches("11pick_kernel") > 0) == pick
        assert (f.launches("13region_kernel") > 0) == (not pick)
        db.close()
