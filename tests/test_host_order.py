"""What the library's host code leaves queued when a call returns, on the fake
runtime: calls that hand out an object work on the legacy stream, which streams
of other calls (non-blocking ones) do not wait for, so none of that work may
be under way when they return."""
import ctypes as C
import os

import numpy as np
import pytest

import kraken2_gb300 as k2g
from fake_cuda import fake_cuda
from kraken_io import GOLDEN

OPTS = k2g.IndexOptions(35, 31, 0, 0xe37e28c4271b5a2d, 1, 1, 0)
PARENT = np.array([0, 0, 1, 1, 2], np.uint64)


@pytest.mark.parametrize("key_bits", [22, 30])      # cells of 32 and 40 bits
def test_a_new_table_is_clear_when_the_call_returns(key_bits):
    with fake_cuda() as f:
        db = k2g.Database.create(OPTS, 1_000_003, key_bits, 10, PARENT)
        assert f.pending() == 0
        db.close()
        assert f.faults() == []


@pytest.mark.parametrize("name", ["db_a", "db_p"])
def test_an_opened_table_is_loaded_when_the_call_returns(name):
    with fake_cuda() as f:
        db = k2g.Database.open(os.path.join(GOLDEN, name))
        assert f.pending() == 0
        n = db.info().node_count
        db.set_names(np.arange(n), [b"x"] * n)
        assert f.pending() == 0
        db.close()
        assert f.faults() == []


def text_reader(db, **kw):
    return k2g.TextReader(db, k2g.ClassifyParams(0.1, 2, 0, 0, 0), chunk_cap=1 << 16, **kw)


def test_a_new_text_reader_leaves_nothing_on_the_legacy_stream():
    """(its per-taxon counts are cleared there or on its own stream, which its
    kernels run on)"""
    with fake_cuda() as f:
        db = k2g.Database.open(os.path.join(GOLDEN, "db_a"))
        t = text_reader(db)
        assert f.pending() == 0
        t.close()
        db.close()
        assert f.faults() == []


def test_new_counters_are_ready_when_the_call_returns():
    with fake_cuda() as f:
        db = k2g.Database.open(os.path.join(GOLDEN, "db_a"))
        c = k2g.Counters(db)
        assert f.pending() == 0
        c.close()
        db.close()
        assert f.faults() == []


def test_merged_replays_start_after_their_flags_have_arrived():
    """The order-exact insert sorts the flagged clusters on the host and sends
    them back: on the stream of the kernel that reads them."""
    with fake_cuda() as f:
        db = k2g.Database.create(OPTS, 100_003, 22, 10, np.array([0, 0, 0, 1, 2], np.uint64))   # two roots
        st = f.stream()
        seen = []

        def launch(name, args):
            def arg(i, ty):
                return C.cast(args[i], C.POINTER(ty))[0]
            if "replay_kernel" in name:          # (view, sorted, n, flags, counter): one flagged cluster
                C.cast(arg(3, C.c_void_p), C.POINTER(C.c_uint64))[0] = 7
                C.cast(arg(4, C.c_void_p), C.POINTER(C.c_uint64))[0] = 1
            if "fixup_kernel" in name:
                seen.append((C.cast(arg(3, C.c_void_p), C.POINTER(C.c_uint64))[0], f.pending()))

        f.hook(launch)
        n = 1000
        db.build_insert(f.device(np.arange(n, dtype=np.uint64)), f.device(np.ones(n, np.uint32)), n, True, st)
        assert seen == [(7, 0)]
        db.close()
        assert f.faults() == []
