"""The warp kernel's list of entries at its size, 320: fragments whose token
groups come to one fewer, as many and one more, once and twice over, against
the oracle."""
import numpy as np
import pytest

import test_gpu_warp as warp
from gpu_util import to_dev, torch

pytestmark = pytest.mark.gpu
ENTRIES = 320


def group_starts(db, seq):
    """For every k-mer of an unambiguous sequence: whether a group starts there
    (its minimizer is not that of the k-mer before)."""
    t = torch()
    mins = t.zeros(len(seq), dtype=t.int64, device="cuda")
    amb = t.zeros(len(seq), dtype=t.uint8, device="cuda")
    d_seq = to_dev(np.concatenate([seq, np.zeros(16, np.uint8)]))
    d_off = to_dev(np.array([0, len(seq)], np.uint64))
    db.scan(d_seq.data_ptr(), d_off.data_ptr(), 1, mins.data_ptr(), amb.data_ptr(),
            t.cuda.current_stream().cuda_stream)
    m = mins.cpu().numpy()[:len(seq) - warp.K + 1]
    return np.concatenate([[True], m[1:] != m[:-1]])


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("paired", [False, True])
def test_fragments_that_fill_the_list(wide, paired):
    db, genome, o = warp.database(wide, False)
    rng = np.random.default_rng(2)
    starts = group_starts(db, genome)
    seqs, counts = [], []
    for target in (ENTRIES - 1, ENTRIES, ENTRIES + 1, 2 * ENTRIES - 1, 2 * ENTRIES, 2 * ENTRIES + 1):
        for at in rng.integers(0, 40_000, 20):
            # the k-mers from `at` on, the first a group's start, up to the target
            upto = np.cumsum(np.concatenate([[True], starts[at + 1:at + 4000]]))
            want = target
            if paired:                          # a mate border between the mates
                want = target - 1 - 50
            n = int(np.searchsorted(upto, want)) + 1 + int(rng.integers(0, 2))
            n = min(n, int(np.searchsorted(upto, want + 1)))
            seqs.append(bytes(genome[at:at + n + warp.K - 1]))
            counts.append(int(upto[n - 1]))
            if paired:
                a2 = int(rng.integers(60_600, 100_000))
                u2 = np.cumsum(np.concatenate([[True], starts[a2 + 1:a2 + 400]]))
                seqs.append(bytes(genome[a2:a2 + int(np.searchsorted(u2, 50)) + warp.K]))
                counts[-1] += 50 + 1
    assert set(counts) == {ENTRIES - 1, ENTRIES, ENTRIES + 1, 2 * ENTRIES - 1, 2 * ENTRIES, 2 * ENTRIES + 1}
    off = np.concatenate([[0], np.cumsum([len(s) for s in seqs])]).astype(np.uint64)
    warp.check(db, o, b"".join(seqs), None, off, len(counts), dict(confidence=0.1, min_hit_groups=2, paired=paired))
