"""Calls of the CUDA runtime that fail, under the library's entry points (on
the fake runtime)."""
import ctypes as C
import os

import numpy as np
import pytest

import kraken2_gb300 as k2g
from fake_cuda import OUT_OF_MEMORY, fake_cuda
from kraken_io import GOLDEN

OPTS = k2g.IndexOptions(35, 31, 0, 0xe37e28c4271b5a2d, 1, 1, 0)
PARENT = np.array([0, 0, 1, 1, 2], np.uint64)
ROOTS = {True: PARENT, False: np.array([0, 0, 0, 1, 2], np.uint64)}
FALLIBLE = ["cudaMallocFromPoolAsync", "cudaMemcpyAsync", "cudaMemsetAsync", "launch", "cudaStreamSynchronize"]


def test_an_error_that_was_reported_is_not_reported_again():
    """The runtime keeps the last error until it is asked for: the check behind
    the next call's first launch must not find it."""
    with fake_cuda() as f:
        db = k2g.Database.create(OPTS, 100_003, 22, 10, PARENT)
        keys, taxa = f.device(np.arange(100, dtype=np.uint64)), f.device(np.ones(100, np.uint32))
        st = f.stream()
        f.fail("cudaMallocFromPoolAsync", 0, OUT_OF_MEMORY)
        with pytest.raises(k2g.K2GError) as e:
            db.build_insert(keys, taxa, 100, False, st)
        assert e.value.status == 5               # K2G_ERR_NOMEM
        db.build_insert(keys, taxa, 100, False, st)
        db.lookup(keys, taxa, 100, st)
        db.close()


def every_failure(f, call, fn, optional=None):
    """call() with the 1st, 2nd ... use of fn failing, until it needs no more."""
    for i in range(400):
        f.fail(fn, i)
        try:
            call()
        except k2g.K2GError:
            assert f.failed(), "an error without a cause"
            assert f.pending_all() == 0, (fn, i)
            continue
        if f.failed():
            # only room asked for ahead of its size, which a build can do without
            assert fn == "cudaMallocFromPoolAsync" and i == optional, (fn, i, "a failure that was not reported")
            continue
        f.fail("", -1)
        return i
    raise AssertionError("too many calls")


def events(f, n):
    """k2g_counters_add's inputs: n events of 40 fragments in two blocks."""
    frags = 40
    d_blocks = f.device((np.arange(frags) // 20).astype(np.uint32))
    reads = k2g.Reads(None, None, None, frags, 0, 0, d_blocks, 0)
    res = k2g.Results()
    res.d_hit_keys, res.d_hit_order = f.device(np.arange(n, dtype=np.uint64)), f.device(np.zeros(n, np.uint64))
    res.d_hit_taxa, res.hits_cap = f.device(np.ones(n, np.uint32)), n
    res.d_hits_used = f.device(np.array([n], np.uint64))
    return reads, res


@pytest.mark.parametrize("fn", FALLIBLE)
@pytest.mark.parametrize("what", ["add", "import", "export", "finish"])
def test_counters(what, fn):
    with fake_cuda() as f:
        db = k2g.Database.create(OPTS, 100_003, 22, 10, PARENT)
        st = f.stream()
        n = 20_000
        state = {"entries": np.arange(n, dtype=np.uint64) << np.uint64(3), "taxon_kmers": np.ones(5, np.uint64),
                 "dense": np.zeros(5, np.uint8)}
        c = k2g.Counters(db)

        def one():
            if what == "add":
                c.add(*events(f, n), stream=st)
            elif what == "import":
                c.import_state(state, stream=st)
            else:
                c.import_state(state, stream=st)
                c.export(st) if what == "export" else c.finish(st)

        every_failure(f, one, fn)
        c.close()
        db.close()
        assert f.faults() == []


@pytest.mark.parametrize("fn", FALLIBLE)
@pytest.mark.parametrize("one_root", [True, False])
@pytest.mark.parametrize("what", ["unordered", "ordered", "sequences", "sample"])
def test_builds(what, one_root, fn):
    with fake_cuda() as f:
        db = k2g.Database.create(OPTS, 100_003, 22, 10, ROOTS[one_root])
        st = f.stream()
        n = 5000
        keys, taxa = f.device(np.arange(n, dtype=np.uint64)), f.device(np.ones(n, np.uint32))
        seq = np.frombuffer(b"ACGT" * 10_000, np.uint8)
        off = np.array([0, 15_000, 40_000], np.uint64)

        def count(name, args):   # (the scan finds a candidate, so that what follows it runs)
            if "block_scan_kernel" in name:
                counts = C.cast(args[5], C.POINTER(C.c_void_p))[0]
                C.cast(counts, C.POINTER(C.c_uint32))[0] = 1

        f.hook(count)

        def one():
            if what == "sequences":
                db.build_sequences(seq, off, np.array([3, 4], np.uint32))
            elif what == "sample":
                db.sample_minimizers(seq, off)
            else:
                db.build_insert(keys, taxa, n, what == "ordered", st)

        # (the seventh allocation of a library scan: bases, chunks, blocks, counts, offsets, sums, then it)
        every_failure(f, one, fn, optional=6 if what in ("sequences", "sample") else None)
        db.close()
        assert f.faults() == []


@pytest.mark.parametrize("fn", ["cudaMalloc", *FALLIBLE, "cudaEventSynchronize"])
def test_text(fn):
    """(the caller's chunk is on its way to the device when the call fails)"""
    with fake_cuda() as f:
        db = k2g.Database.create(OPTS, 100_003, 22, 10, PARENT)
        n = 100
        chunk = b"".join(b"@r%d\n%s\n+\n%s\n" % (i, b"ACGT" * 30, b"I" * 120) for i in range(n))

        def launch(name, args):      # what the parser finds: the whole chunk's records, one block
            if "11frag_kernel" in name:
                info = C.cast(C.cast(args[5], C.POINTER(C.c_void_p))[0], C.POINTER(C.c_uint64))
                for word, value in ((0, 2**64 - 1), (1, 120), (2, n), (3, n), (4, 1), (5, len(chunk)), (6, 120 * n)):
                    info[word] = value

        f.hook(launch)
        t = k2g.TextReader(db, k2g.ClassifyParams(0.1, 2, 0, 0, 0), chunk_cap=1 << 16, lines=False)
        counters = k2g.Counters(db)

        def one():
            t.reset()
            res, _ = t.classify(chunk, True, counters)
            assert (res.fragments, res.handoff) == (n, 0)

        every_failure(f, one, fn)
        t.close()
        counters.close()
        db.close()
        assert f.faults() == []


MAKING = ["cudaMalloc", "cudaMallocFromPoolAsync", "cudaMemcpy", "cudaMemset", "cudaMemcpyAsync", "cudaMemsetAsync",
          "launch", "cudaStreamSynchronize", "cudaEventRecord", "cudaEventSynchronize", "cudaStreamCreate",
          "cudaStreamCreateWithFlags", "cudaHostAlloc", "cudaEventCreateWithFlags"]


def every_failure_in_making(f, make):
    """make() with each call of the runtime failing in turn: it says so, and
    keeps no memory."""
    for fn in MAKING:
        for i in range(200):
            held = f.used()
            f.fail(fn, i)
            try:
                made = make()
            except k2g.K2GError:
                assert f.failed() and f.used() == held, (fn, i)
                continue
            assert not f.failed(), (fn, i, "a failure that was not reported")
            f.fail("", -1)
            made.close()
            assert f.used() == held, fn
            break
        else:
            raise AssertionError("too many calls")
    assert f.faults() == []


@pytest.mark.parametrize("key_bits", [22, 30])
def test_tables(key_bits):
    with fake_cuda() as f:
        every_failure_in_making(f, lambda: k2g.Database.create(OPTS, 100_003, key_bits, 10, PARENT))


def test_opened_tables():
    with fake_cuda() as f:
        every_failure_in_making(f, lambda: k2g.Database.open(os.path.join(GOLDEN, "db_a")))


@pytest.mark.parametrize("what", ["counters", "text", "server"])
def test_objects(what):
    with fake_cuda() as f:
        db = k2g.Database.open(os.path.join(GOLDEN, "db_a"))
        cp = k2g.ClassifyParams(0.1, 2, 0, 0, 0)
        make = {"counters": lambda: k2g.Counters(db), "text": lambda: k2g.TextReader(db, cp, chunk_cap=1 << 16),
                "server": lambda: k2g.Server(db, cp, 64 << 20)}[what]
        make().close()               # (the pool's stream)
        every_failure_in_making(f, make)
        db.close()
