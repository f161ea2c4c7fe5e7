"""k2g_classify under stream capture: the one-launch form, which allocates
nothing, and the pieces form, whose allocation becomes part of the graph.  The
graph is launched again on other reads in the same buffers, with calls outside
it in between, and gives what k2g_classify gives."""
import numpy as np
import pytest

import kraken2_gb300 as k2g
import test_gpu_warp as warp
from gpu_util import bytes_dev, to_dev, torch, u32, u64, zeros

pytestmark = pytest.mark.gpu


def outputs(t, n, cap, nodes):
    return dict(call=zeros(n, t.int32), hg=zeros(n, t.int32), hoff=zeros(n, t.int64), hlen=zeros(n, t.int32),
                runs=zeros(cap, t.int64), tr=zeros(nodes, t.int64), status=zeros(1, t.int32))


def results(o, cap):
    return k2g.Results(o["call"].data_ptr(), o["hg"].data_ptr(), o["hoff"].data_ptr(), o["hlen"].data_ptr(),
                       o["runs"].data_ptr(), cap, o["tr"].data_ptr(), None, None, None, 0, None, o["status"].data_ptr())


def lists(o, n):
    """Every output of the call, the runs fragment by fragment."""
    hoff, hlen, runs = u64(o["hoff"]), u32(o["hlen"]), u64(o["runs"])
    flat = [runs[int(a):int(a) + int(m)] for a, m in zip(hoff[:n], hlen[:n])]
    return [u32(o["call"])[:n], u32(o["hg"])[:n], hlen[:n], np.concatenate(flat), u64(o["tr"]), u32(o["status"])]


@pytest.mark.parametrize("lens", [[150] * 3000, [30, 5000, 300, 20_000, 4096, 0, 8191] * 20], ids=["short", "pieces"])
def test_a_captured_call_is_replayed(lens):
    t = torch()
    db, genome, _ = warp.database(False, False)
    nodes, n = int(db.info().node_count), len(lens)
    made = [warp.batch(genome, lens, seed) for seed in (1, 2, 3)]
    off = made[0][2]
    cap = int(off[-1]) + 2 * n + 8
    d_bases, d_off = bytes_dev(made[0][0]), to_dev(off)
    reads = k2g.Reads(d_bases.data_ptr(), None, d_off.data_ptr(), n, max(lens), int(off[-1]), None, 0)
    cp = k2g.ClassifyParams(0.05, 2, 0, 0, 0)

    def plain():
        o = outputs(t, n, cap, nodes)
        db.classify(reads, cp, results(o, cap), mode=k2g.MODE_PIPELINED, stream=t.cuda.current_stream().cuda_stream)
        t.cuda.synchronize()
        return lists(o, n)

    plain()                                      # (the module and the pool are there before the capture)
    o = outputs(t, n, cap, nodes)
    g, st = t.cuda.CUDAGraph(), t.cuda.Stream()
    t.cuda.synchronize()
    with t.cuda.graph(g, stream=st):
        db.classify(reads, cp, results(o, cap), mode=k2g.MODE_PIPELINED, stream=st.cuda_stream)
    t.cuda.synchronize()
    assert not o["call"].any()                   # (captured, not run)
    for bases, _, other in made * 2:
        assert np.array_equal(other, off)
        d_bases[:len(bases)] = bytes_dev(bases)[:len(bases)]
        o["tr"].zero_()
        want = plain()
        g.replay()
        t.cuda.synchronize()
        for a, b in zip(lists(o, n), want):
            assert np.array_equal(a, b)
    assert want[0].any()
