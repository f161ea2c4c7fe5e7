"""Which kernels take a call (on the fake runtime).  ResolveTree joins the taxa
of the highest score by LCA one after another; where a taxonomy has several
roots an LCA can be 0, and LCA(0, x) is x, so the result is not the ancestor of
all of them, which is what the warp kernels look for.  Such tables keep the
kernels that join one by one."""
import numpy as np
import pytest

import kraken2_gb300 as k2g
from fake_cuda import fake_cuda

ONE_ROOT = np.array([0, 0, 1, 1, 2, 2], np.uint64)
TWO_ROOTS = np.array([0, 0, 1, 0, 2, 3], np.uint64)


@pytest.mark.parametrize("k,l,dna,kernel,staged", [(35, 31, 1, "warp_classify_kernel", "pipe_step_kernel"),
                                                   (15, 12, 0, "warp_translated_kernel", "17translated_kernel")])
@pytest.mark.parametrize("parent", [ONE_ROOT, TWO_ROOTS], ids=["one root", "two roots"])
def test_tables_with_several_roots_are_resolved_one_by_one(parent, k, l, dna, kernel, staged):
    with fake_cuda() as f:
        db = k2g.Database.create(k2g.IndexOptions(k, l, 0, 0, dna, 1, 0), 100_003, 22, 10, parent, device=57)
        n, length = 10, 150
        out = f.device(np.zeros(n * length + 64, np.uint64))
        off = f.device(np.arange(n + 1, dtype=np.uint64) * np.uint64(length))
        reads = k2g.Reads(f.device(np.zeros(n * length, np.uint8)), None, off, n, length, n * length, None, 0)
        res = k2g.Results(out, None, None, None, out, n * length + 32, None, None, None, None, 0, None, out)
        db.classify(reads, k2g.ClassifyParams(0.0, 2, 0, 0, 0), res, mode=k2g.MODE_PIPELINED, stream=f.stream())
        one = parent is ONE_ROOT
        assert (f.launches(kernel) > 0) == one and (f.launches(staged) > 0) == (not one)
        db.close()
