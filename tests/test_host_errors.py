"""Calls of the CUDA runtime that fail, under the library's entry points (on
the fake runtime)."""
import numpy as np
import pytest

import kraken2_gb300 as k2g
from fake_cuda import fake_cuda

OPTS = k2g.IndexOptions(35, 31, 0, 0xe37e28c4271b5a2d, 1, 1, 0)
PARENT = np.array([0, 0, 1, 1, 2], np.uint64)


def test_an_error_that_was_reported_is_not_reported_again():
    """The runtime keeps the last error until it is asked for: the check behind
    the next call's first launch must not find it."""
    with fake_cuda() as f:
        db = k2g.Database.create(OPTS, 100_003, 22, 10, PARENT)
        keys, taxa = f.device(np.arange(100, dtype=np.uint64)), f.device(np.ones(100, np.uint32))
        st = f.stream()
        f.fail("cudaMallocFromPoolAsync", 0)
        with pytest.raises(k2g.K2GError) as e:
            db.build_insert(keys, taxa, 100, False, st)
        assert e.value.status == 5               # K2G_ERR_NOMEM
        db.build_insert(keys, taxa, 100, False, st)
        db.lookup(keys, taxa, 100, st)
        db.close()
