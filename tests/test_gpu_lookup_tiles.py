"""k2g_lookup at the edges of its tiles, on tables within and beyond L2, with
walks that leave their sector, wrap around and meet the partial last one."""
import numpy as np
import pytest

import kraken2_gb300 as k2g
import oracle
from gpu_util import to_dev, torch, u32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("capacity,load,n", [(11, 1.0, 1), (1003, 1.0, 255), (1003, 0.97, 257), (100_003, 0.9, 768),
                                             (100_003, 0.7, 1_000_003), (35_000_003, 0.7, 300_001)])
def test_lookups_equal_the_oracle(capacity, load, n, wide):
    t = torch()
    rng = np.random.default_rng(n)
    nodes = 1000
    parent = np.concatenate([[0], np.arange(nodes - 1) // 2]).astype(np.uint64)
    kb = 30 if wide else 22
    db = k2g.Database.create(k2g.IndexOptions(35, 31, 0, 0, 1, 1, 0), capacity, kb, 10, parent)
    stored = rng.integers(0, 2**62, int(capacity * load), dtype=np.int64).astype(np.uint64)
    taxa = rng.integers(1, nodes, len(stored)).astype(np.uint32)
    d_stored, d_taxa = to_dev(stored), to_dev(taxa)
    db.build_insert(d_stored.data_ptr(), d_taxa.data_ptr(), len(stored), False, t.cuda.current_stream().cuda_stream)
    keys = np.where(rng.random(n) < 0.6, stored[rng.integers(0, len(stored), n)],
                    rng.integers(0, 2**62, n, dtype=np.int64).astype(np.uint64))
    d_keys = to_dev(keys)
    vals = t.zeros(n, dtype=t.int32, device="cuda")
    db.lookup(d_keys.data_ptr(), vals.data_ptr(), n, t.cuda.current_stream().cuda_stream)
    cells, _ = db.download()
    o = oracle.Oracle(cells, capacity, kb, 10, parent, oracle.index_opts(35, 31, 0, 0))
    if wide:   # (the oracle's batch lookup reads 32-bit cells: a plain walk here)
        c = np.zeros((capacity, 8), np.uint8)
        c[:, :5] = cells.reshape(-1, 5)
        c = c.view(np.uint64).reshape(-1)
        from bench import murmur3_np
        hc = murmur3_np(keys)
        want = np.zeros(n, np.uint32)
        for i in range(min(n, 20_000)):
            at = first = int(hc[i]) % capacity
            while True:
                cell = int(c[at])
                if not cell & 1023:
                    break
                if ((cell >> 10) & 0xFFFFFFFF) == int(hc[i]) >> (64 - kb):
                    want[i] = cell & 1023
                    break
                at = (at + 1) % capacity
                if at == first:
                    break
        m = min(n, 20_000)
        assert np.array_equal(u32(vals)[:m], want[:m])
    else:
        assert np.array_equal(u32(vals), o.get_batch(keys, threads=8))
    db.close()
