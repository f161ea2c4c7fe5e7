"""The buffers that k2g_classify_host keeps between calls, on the fake runtime:
after an allocation that failed, the next call, of any size, finds buffers that
are as large as it takes them to be."""
import ctypes as C

import numpy as np
import pytest

import kraken2_gb300 as k2g
from fake_cuda import fake_cuda

OPTS = k2g.IndexOptions(35, 31, 0, 0xe37e28c4271b5a2d, 1, 1, 0)
PARENT = np.array([0, 0, 1, 1, 2], np.uint64)


def classify(db, n, length=150, counters=None, quals=True, nodes=len(PARENT)):
    bases = np.full(n * length + 16, ord("A"), np.uint8)
    off = np.arange(n + 1, dtype=np.uint64) * np.uint64(length)
    call, hg, hlen = (np.zeros(n, np.uint32) for _ in range(3))
    runs, tr = np.zeros(16, np.uint64), np.zeros(nodes, np.uint64)
    nr = C.c_uint64(len(runs))
    cp = k2g.ClassifyParams(0.0, 2, 0, 0, 10)
    args = [db.h, bases.ctypes.data, bases.ctypes.data if quals else None, off.ctypes.data, n]
    out = [C.byref(cp), call.ctypes.data, hg.ctypes.data, hlen.ctypes.data, runs.ctypes.data, C.byref(nr),
           tr.ctypes.data]
    if counters is None:
        return k2g.lib().k2g_classify_host(*args, *out)
    blocks = (np.arange(n) // 100).astype(np.uint32)
    return k2g.lib().k2g_classify_host_blocks(*args, blocks.ctypes.data, counters.h, *out)


@pytest.mark.parametrize("with_counters", [False, True])
def test_a_failed_allocation_leaves_no_capacity_behind(with_counters):
    with fake_cuda() as f:
        small = k2g.Database.create(OPTS, 100_003, 22, 10, PARENT, device=11 + with_counters)
        large = k2g.Database.create(OPTS, 100_003, 22, 10, np.arange(1000, dtype=np.uint64) // 2, device=11 + with_counters)
        cs = [k2g.Counters(db) if with_counters else None for db in (small, large)]
        n = 500
        for i in range(60):
            k2g.check(classify(small, n, counters=cs[0]))
            n += 50                                  # every buffer has to grow
            f.fail("cudaMalloc", i)
            status = classify(large, n, counters=cs[1], nodes=1000)
            assert (status != 0) == f.failed()
            f.fail("", -1)
            k2g.check(classify(small, 500, counters=cs[0]))
            k2g.check(classify(large, 500, counters=cs[1], nodes=1000))
            assert f.faults() == []
            if status == 0:
                break
        assert status == 0 and i > 10


@pytest.mark.parametrize("fn", ["cudaMalloc", "cudaHostAlloc", "cudaStreamCreateWithFlags",
                                "cudaStreamCreateWithPriority", "cudaEventCreateWithFlags"])
def test_a_first_call_that_failed_half_way(fn):
    with fake_cuda() as f:
        # (a device of its own for each of the calls made to fail)
        first = 20 + 8 * ["cudaHostAlloc", "cudaStreamCreateWithFlags", "cudaStreamCreateWithPriority",
                          "cudaEventCreateWithFlags", "cudaMalloc"].index(fn)
        for i in range(8):
            db = k2g.Database.create(OPTS, 100_003, 22, 10, PARENT, device=first + i)
            f.fail(fn, i)
            status = classify(db, 500)
            assert (status != 0) == f.failed()
            f.fail("", -1)
            k2g.check(classify(db, 500))
            k2g.check(classify(db, 700))
            db.close()
            assert f.faults() == []
            if status == 0:
                break
        assert i > 0


def staged_call(f, db, st, n, events):
    """k2g_classify of n fragments of 150 bases; whether it succeeded."""
    bases = f.device(np.full(150 * n, ord("A"), np.uint8))
    off = f.device(np.arange(n + 1, dtype=np.uint64) * np.uint64(150))
    out = f.device(np.zeros(400 * n, np.uint64))
    reads = k2g.Reads(bases, None, off, n, 150, 150 * n, None, 0)
    res = k2g.Results(out, None, None, None, out, 152 * n, None, out if events else None, out, out, n, out, out)
    try:
        db.classify(reads, k2g.ClassifyParams(0.0, 2, 0, 0, 0), res, mode=k2g.MODE_PIPELINED, stream=st)
        return True
    except k2g.K2GError:
        return False
    finally:
        for p in (bases, off, out):
            f.lib.cudaFree(C.c_void_p(p))


def test_staged_buffers_after_a_failed_allocation():
    """k2g_classify on a table that the staged kernels take (k = l): whatever
    failed in between, a call's kernels get every pointer they got before."""
    with fake_cuda() as f:
        db = k2g.Database.create(k2g.IndexOptions(31, 31, 0, 0xe37e28c4271b5a2d, 1, 1, 0), 100_003, 22, 10, PARENT,
                                 device=61)
        st = f.stream()

        def call(n, events):
            return staged_call(f, db, st, n, events)

        given = []

        def launch(name, args):              # which words of a launch's argument are null
            if "pipe_step_kernel" in name:
                words = C.cast(args[0], C.POINTER(C.c_uint64))[:128]
                given.append([w != 0 for w in words])

        f.hook(launch)
        assert call(1000, True) and call(1000, True)
        want = given[len(given) // 2:]
        n = 1000
        for i in range(60):
            n += 500
            f.fail("cudaMalloc", i + 3)          # (three are the caller's)
            done = call(n, True)
            assert done != f.failed()
            f.fail("", -1)
            given.clear()
            assert call(1000, True) and given == want
            if done:
                break
        assert done and i > 3


def test_staged_hit_keys_have_room_for_every_slot():
    """A call with hit events behind a larger one without: the slots are still
    those of the larger one."""
    with fake_cuda() as f:
        db = k2g.Database.create(k2g.IndexOptions(31, 31, 0, 0xe37e28c4271b5a2d, 1, 1, 0), 100_003, 22, 10, PARENT,
                                 device=62)
        st = f.stream()
        seen = []

        def launch(name, args):
            if "pipe_step_kernel" in name:       # the scan role's view: its last two words
                gkey, cap_slots = C.cast(args[0], C.POINTER(C.c_uint64))[58:60]
                seen.append((f.room(gkey), 8 * cap_slots))

        assert staged_call(f, db, st, 20_000, False)
        f.hook(launch)
        assert staged_call(f, db, st, 1000, True)
        assert seen and all(have >= need > 0 for have, need in seen)


@pytest.mark.parametrize("with_counters", [False, True])
@pytest.mark.parametrize("length", [150, 5000])      # three slots, and four for long fragments
def test_a_device_with_room_for_two_slots(length, with_counters):
    """Calls of several chunks take more slots than two for speed alone: where
    memory is short, two do, also when others hold some from an earlier call."""
    with fake_cuda() as f:
        n = (400 << 20 if with_counters else 130 << 20) // length        # five chunks and more
        slots = 4 if length == 5000 and not with_counters else 3

        def call(db, frags):
            c = k2g.Counters(db) if with_counters else None
            return classify(db, frags, length, c, quals=False)

        first = 30 + 6 * (length == 5000) + 3 * with_counters            # (devices of their own)
        dbs = [k2g.Database.create(OPTS, 100_003, 22, 10, PARENT, device=first + i) for i in range(3)]
        base = f.used()
        k2g.check(call(dbs[0], n))
        slot = (f.used() - base) // slots
        base = f.used()
        f.limit(base + 5 * slot // 2)
        k2g.check(call(dbs[1], n // 2))                                  # (fewer, or smaller, chunks)
        for _ in range(2):
            k2g.check(call(dbs[1], n))
        f.limit(1 << 60)
        k2g.check(call(dbs[1], n))
        # with room for one there is an error, which leaves the next call whole
        base = f.used()
        f.limit(base + 3 * slot // 2)
        assert call(dbs[2], n) == 5
        f.limit(1 << 60)
        k2g.check(call(dbs[2], n))
        assert f.faults() == []


@pytest.mark.parametrize("what", ["table", "wide table", "host", "staged", "text", "server", "lines"])
def test_memory_that_the_pool_keeps_is_there_for_others(what):
    """(up to 1 GB, which a program that needs it for a table or a call gets)"""
    with fake_cuda() as f:
        staged = k2g.IndexOptions(31, 31, 0, 0xe37e28c4271b5a2d, 1, 1, 0)
        roots = np.array([0, 0, 0, 1, 2], np.uint64)             # (an ordered insert sorts all pairs)
        db = k2g.Database.create(staged if what == "staged" else OPTS, 100_003, 22, 10, roots, device=63)
        if what in ("text", "lines"):
            db.set_names(np.arange(5), [b"x"] * 5)
        n = 20_000_000
        keys, taxa = f.device(np.zeros(n, np.uint64)), f.device(np.zeros(n, np.uint32))
        db.build_insert(keys, taxa, n, True, f.stream())
        assert f.kept() > 100 << 20
        cp = k2g.ClassifyParams(0.0, 2, 0, 0, 0)

        def call():
            if what == "table":
                k2g.Database.create(OPTS, 40_000_003, 22, 10, PARENT, device=63).close()
            elif what == "wide table":
                k2g.Database.create(OPTS, 20_000_003, 30, 10, PARENT, device=63).close()
            elif what == "host":
                k2g.check(classify(db, 5000, quals=False))
            elif what == "staged":
                assert staged_call(f, db, f.stream(), 2000, False)
            elif what == "text":
                k2g.TextReader(db, cp, chunk_cap=1 << 20).close()
            elif what == "server":
                k2g.Server(db, cp, 64 << 20).close()
            else:
                m = 1_000_000
                db.format_lines(np.zeros(m, np.uint32), np.zeros(m, np.uint32), np.zeros(0, np.uint64), [b"r"] * m,
                                np.full(m, 150))

        f.limit(f.used() + f.kept() + (16 << 20))    # (the call needs more than that, and less than what is kept)
        call()
        assert f.kept() < 100 << 20 and f.faults() == []
        f.limit(1 << 60)
        db.close()
