"""What the library's host code leaves queued when a call returns, on the fake
runtime: calls that hand out an object work on the legacy stream, which streams
of other calls (non-blocking ones) do not wait for, so none of that work may
be under way when they return."""
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
