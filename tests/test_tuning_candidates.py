"""k2g_autotune times a form of the call only once, and every form that the
values can give it: its calls are counted on the fake runtime, where all take
the same time and so the first, the table's defaults, is kept."""
import numpy as np
import pytest

import kraken2_gb300 as k2g
from fake_cuda import fake_cuda

PARENT = np.array([0, 0, 1, 1, 2], np.uint64)
TRIALS = 3


def autotune(f, db, length, n=64, paired=False, quick=False):
    """(launches of the calls' main kernels, the values kept and the defaults)"""
    per = 2 if paired else 1
    off = np.arange(n * per + 1, dtype=np.uint64) * np.uint64(length)
    total = int(off[-1])
    out = f.device(np.zeros(total + 2 * n + 16, np.uint64))
    reads = k2g.Reads(f.device(np.zeros(total, np.uint8)), None, f.device(off), n, length, total, None, 0)
    res = k2g.Results(out, None, None, None, out, total + 2 * n + 8, None, None, None, None, 0, None, out)
    cls = k2g.length_class(total, n)
    default = db.tuning(paired, cls).as_dict()
    before = {k: f.launches(k) for k in KERNELS}
    chosen, _ = db.autotune(reads, k2g.ClassifyParams(0.0, 2, int(quick), int(paired), 0), res, trials=TRIALS,
                            stream=f.stream())
    assert db.tuning(paired, cls).as_dict() == chosen.as_dict()
    return {k: f.launches(k) - before[k] for k in KERNELS}, chosen.as_dict(), default


KERNELS = ["warp_classify_kernel", "warp_translated_kernel", "warp_merge_kernel", "pipe_step_kernel"]
ONE = 1 + TRIALS                      # calls of a candidate


# pieces of 1,024, 2,048, 4,096 and 8,192 bases cut reads twice as long and
# more; a form that cuts nothing is one more, where there is one
@pytest.mark.parametrize("length,forms,cutting", [(150, 1, 0), (2047, 1, 0), (2048, 2, 1), (4096, 3, 2), (8192, 4, 3),
                                                  (16383, 4, 3), (16384, 4, 4), (100_000, 4, 4)])
def test_one_call_a_form_on_default_tables(length, forms, cutting):
    with fake_cuda() as f:
        db = k2g.Database.create(k2g.IndexOptions(35, 31, 0, 0, 1, 1, 0), 100_003, 22, 10, PARENT, device=50)
        launches, chosen, default = autotune(f, db, length)
        # (the last call is the one that leaves the outputs, with the defaults)
        assert launches["warp_classify_kernel"] == ONE * forms + 1
        assert launches["warp_merge_kernel"] == ONE * cutting + (length >= 8 * default["piece_len"])
        assert launches["pipe_step_kernel"] == 0 and chosen == default
        db.close()


@pytest.mark.parametrize("how", [dict(paired=True), dict(quick=True)])
def test_pairs_and_quick_calls_have_one_form(how):
    with fake_cuda() as f:
        db = k2g.Database.create(k2g.IndexOptions(35, 31, 0, 0, 1, 1, 0), 100_003, 22, 10, PARENT, device=50)
        launches, chosen, default = autotune(f, db, 20_000, **how)
        assert launches["warp_classify_kernel"] == ONE + 1 and chosen == default
        db.close()


def test_translated_search_has_one_form():
    with fake_cuda() as f:
        db = k2g.Database.create(k2g.IndexOptions(15, 12, 0, 0, 0, 1, 0), 100_003, 22, 10, PARENT, device=50)
        launches, chosen, default = autotune(f, db, 150)
        assert launches["warp_translated_kernel"] == ONE + 1 and chosen == default
        db.close()


def test_other_tables_keep_the_staged_candidates():
    with fake_cuda() as f:
        db = k2g.Database.create(k2g.IndexOptions(31, 31, 0, 0, 1, 1, 0), 100_003, 22, 10, PARENT, device=50)
        launches, chosen, _ = autotune(f, db, 150)
        # three probe splits and four sub-batch sizes, one sub-batch each: three beats
        assert launches["pipe_step_kernel"] >= 3 * 12 * ONE
        db.close()
