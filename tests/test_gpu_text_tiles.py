"""The text path at the edges of its line tiles (1,024 lines) and window
tiles (16 KB): lines just below, at and above them, a damaged line on either
side, more lines than the buffers hold, and kraken lines that fit a warp's
stage (4 KB) or not."""
import numpy as np
import pytest

import kraken2_gb300 as k2g
from test_gpu_text import cparams, expected_lines, gpu_db, run_text, synth_reads

pytestmark = pytest.mark.gpu

DEFAULT = dict(confidence=0.0, min_hit_groups=2, quick=False, paired=False, min_quality=0)


def reader(cap):
    return k2g.TextReader(gpu_db("db_a"), cparams(DEFAULT), chunk_cap=cap, block_bytes=3 << 20)


def records(n, kind, rng, lo, hi):
    out = []
    for i, s in enumerate(synth_reads(rng, n, lo, hi)):
        seq = s if isinstance(s, bytes) else s[1]
        if kind == "fastq":
            out.append(b"@r%d x\n%s\n+\n%s\n" % (i, seq, b"I" * len(seq)))
        else:
            cut = len(seq) // 2
            out.append(b">r%d\n%s\n%s\n" % (i, seq[:cut], seq[cut:]))
    return out


@pytest.mark.parametrize("kind", ["fastq", "fasta"])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 341, 342, 683, 1024, 3000])
@pytest.mark.parametrize("lo,hi", [(40, 120), (300, 3000)])
def test_records_around_line_tiles(kind, n, lo, hi):
    rng = np.random.default_rng(n + lo)
    recs = records(n, kind, rng, lo, hi)
    data = b"".join(recs)
    tr = reader(max(len(data), 4096))
    text, frags, _, handoff = run_text(tr, data, len(data))
    assert handoff is None and frags == n
    assert text == expected_lines("db_a", data, DEFAULT)
    # a damaged record at a tile's edges: everything before it is classified
    # when it starts a reader block (blocks of one record here)
    tr.close()
    if n < 256:
        return
    tr = k2g.TextReader(gpu_db("db_a"), cparams(DEFAULT), chunk_cap=len(data) + 64, block_bytes=1)
    per = 4 if kind == "fastq" else 3
    for at in {1023 // per, 1024 // per, min(1025 // per + 1, n - 1), n - 1}:
        if at >= n:
            continue
        bad = recs[at].replace(b"\n+\n", b"\n-\n") if kind == "fastq" else recs[at][:-1] + b"\n+\n"
        dam = b"".join(recs[:at]) + bad + b"".join(recs[at + 1:])
        text, frags, _, handoff = run_text(tr, dam, len(dam))
        assert handoff == sum(len(r) for r in recs[:at]) and frags == at
        assert text == expected_lines("db_a", b"".join(recs[:at]), DEFAULT, block_bytes=1)
    tr.close()


def test_too_many_lines_are_handed_back():
    data = b">a\n" + b"A\n" * 40_000
    tr = reader(len(data))
    text, frags, _, handoff = run_text(tr, data, len(data))
    assert (text, frags, handoff) == (b"", 0, 0)
    # the reader works on afterwards
    ok = b">b\n" + b"ACGT" * 30 + b"\n"
    text, frags, _, handoff = run_text(tr, ok, len(ok))
    assert handoff is None and text == expected_lines("db_a", ok, DEFAULT)
    tr.close()
