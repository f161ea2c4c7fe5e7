"""The work that programs have this library do, at the sizes they meet.

Every case goes through the public entry points (the Python mirror of the C
ABI): classification of reads held on the device, of reads in host memory, of
FASTQ text, with minimizer counters, against a protein table; batched table
lookups; and a library build.  Tables, genomes and reads are synthetic and
follow from the seed: genomes are uniform random sequence or families of
related strains, their minimizers are inserted order-exact (so the table does
not depend on thread timing), the rest of a table is filled with random keys
to a load of 0.7, and reads are stretches of the genomes with substitutions,
or random sequence.
"""
import ctypes as C
import math

import numpy as np
import torch

import kraken2_gb300 as k2g

K, L_MER = 35, 31                     # nucleotide defaults: k, l, 7 spaced positions
SEED_TEMPLATE = "1" * 17 + "01" * 7
TOGGLE = 0xE37E28C4271B5A2D
PROTEIN_K, PROTEIN_L = 15, 12
LOAD = 0.7
BLOCK_BASES = 3 * 1024 * 1024         # reader blocks of single reads
STRAINS, SPECIES = 4, 4               # strains per species, species per genus

# What each case stands for:
#   kind "device"      k2g_classify on reads resident in HBM, as a program does
#                      that reads and batches by itself
#   kind "host"        k2g_classify_host: reads and results in (pinned) host memory
#   kind "text"        k2g_text_*: FASTQ bytes in, kraken lines out, the path of
#                      the classify executable
#   kind "counters"    k2g_classify_host_blocks with -K counters, and the finish
#   kind "translated"  k2g_classify on a protein table (six frames)
#   kind "lookup"      k2g_lookup: the batched form of the reference's table Get
#   kind "build"       an empty table and k2g_build_sequences (order-exact build)
_DEVICE = {"kind": "device", "paired": False, "quality": 0, "quick": False, "wide": False,
           "related": False, "confidence": 0.0, "n_rate": 0.0}


def listed():
    return [
        # one small request, a table that fits L2: launches and latency count
        {**_DEVICE, "name": "call_1k", "reads": 1000, "len_min": 150, "len_max": 150,
         "cells": 2_275_497},
        # a reader block's worth of trimmed reads of uneven length with N bases and
        # quality masking (-Q)
        {**_DEVICE, "name": "ragged_20k_quality", "reads": 20_011, "len_min": 30, "len_max": 301,
         "cells": 24_000_001, "quality": 20, "n_rate": 0.002, "related": True},
        # the standard batch of an 8M-read call against a table of 16 GB
        {**_DEVICE, "name": "short_8m", "reads": 8_000_000, "len_min": 150, "len_max": 150,
         "cells": 4_000_000_000, "confidence": 0.1},
        # pairs from related genomes, with a confidence threshold: several taxa a read
        {**_DEVICE, "name": "pairs_500k", "reads": 500_000, "len_min": 150, "len_max": 150,
         "cells": 250_000_007, "paired": True, "related": True, "confidence": 0.1},
        # quick mode against a table of 40-bit cells
        {**_DEVICE, "name": "quick_wide_300k", "reads": 300_000, "len_min": 250, "len_max": 250,
         "cells": 100_000_007, "quick": True, "wide": True},
        # short reads in host memory, results back in host memory
        {"name": "host_2m", "kind": "host", "reads": 2_000_000, "long_reads": 0, "length": 150,
         "cells": 500_000_000, "related": False, "confidence": 0.1},
        # one long read (log-normal, mean 5 kb, up to 50 kb) to five of 150 bp
        {"name": "host_long_mix", "kind": "host", "reads": 100_000, "long_reads": 20_000,
         "length": 150, "cells": 500_000_000, "related": True, "confidence": 0.1},
        # 128 MB of FASTQ in 32 MB chunks
        {"name": "fastq_404k", "kind": "text", "reads": 404_000, "length": 150, "chunk": 32 << 20,
         "cells": 500_000_000, "related": False, "confidence": 0.1},
        # --report-minimizer-data over a sample of a million reads
        {"name": "minimizer_data_1m", "kind": "counters", "reads": 1_000_000, "length": 150,
         "cells": 500_000_000, "related": True, "confidence": 0.1},
        # translated search
        {"name": "translated_100k", "kind": "translated", "reads": 100_000, "length": 150,
         "residues": 4_000_000},
        # keys of a CPU caller's batch, looked up on the device
        {"name": "lookup_16m", "kind": "lookup", "keys": 16_777_213, "cells": 500_000_000},
        # a library of 48 Mbp added to a new table
        {"name": "build_48mbp", "kind": "build", "bases": 48_000_000, "genomes": 480,
         "cells": 24_000_001},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["device"] * 5 + ["host", "host", "text", "counters", "translated", "lookup", "build"])
    cells = _log_uniform(rng, 1 << 19, 1_000_000_000) | 1
    if kind == "device":
        hi = rng.choice([rng.randint(50, 151), rng.randint(100, 301), rng.randint(200, 500)])
        lo = rng.choice([hi, hi, rng.randint(20, hi)])
        paired = rng.random() < 0.35
        reads = _log_uniform(rng, 300, 1_200_000_000 // (hi * (4 if paired else 2)))
        return {**_DEVICE, "reads": reads, "len_min": lo, "len_max": hi, "cells": cells,
                "paired": paired, "quality": rng.choice([0, 0, 0, 10, 20]),
                "quick": rng.random() < 0.15, "wide": rng.random() < 0.15,
                "related": rng.random() < 0.5, "confidence": rng.choice([0.0, 0.05, 0.1, 0.5]),
                "n_rate": rng.choice([0.0, 0.001, 0.01])}
    if kind == "host":
        long_reads = rng.choice([0, _log_uniform(rng, 20, 20_000)])
        return {"kind": kind, "reads": _log_uniform(rng, 1000, 500_000), "long_reads": long_reads,
                "length": rng.randint(75, 251), "cells": cells, "related": rng.random() < 0.5,
                "confidence": rng.choice([0.0, 0.1])}
    if kind == "text":
        return {"kind": kind, "reads": _log_uniform(rng, 2000, 400_000), "length": rng.randint(75, 251),
                "chunk": rng.choice([8 << 20, 32 << 20, 64 << 20]), "cells": cells,
                "related": rng.random() < 0.5, "confidence": rng.choice([0.0, 0.1])}
    if kind == "counters":
        return {"kind": kind, "reads": _log_uniform(rng, 20_000, 1_000_000),
                "length": rng.randint(75, 251), "cells": cells, "related": rng.random() < 0.5,
                "confidence": rng.choice([0.0, 0.1])}
    if kind == "translated":
        return {"kind": kind, "reads": _log_uniform(rng, 1000, 200_000),
                "length": rng.randint(75, 301), "residues": _log_uniform(rng, 200_000, 8_000_000)}
    if kind == "lookup":
        return {"kind": kind, "keys": _log_uniform(rng, 1000, 40_000_000), "cells": cells}
    bases = _log_uniform(rng, 1_000_000, 64_000_000)
    return {"kind": kind, "bases": bases, "genomes": rng.choice([16, 64, 256, 480]),
            "cells": int(bases / 2) | 1}


# ---- inputs -----------------------------------------------------------------

def _spaced_mask():
    out = 0
    for bit in SEED_TEMPLATE:
        out = (out << 2) | (3 if bit == "1" else 0)
    return out


def _options(protein=False):
    if protein:
        return k2g.IndexOptions(PROTEIN_K, PROTEIN_L, 0, TOGGLE, 0, 1, 0)
    return k2g.IndexOptions(K, L_MER, _spaced_mask(), TOGGLE, 1, 1, 0)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _taxonomy(genomes):
    """root 1, genera, species, one strain per genome (parent < child);
    returns (parents, taxon of every genome)."""
    n_sp = -(-genomes // STRAINS)
    n_ge = -(-n_sp // SPECIES)
    first_sp, first_st = 2 + n_ge, 2 + n_ge + n_sp
    parent = np.zeros(first_st + genomes, np.uint64)
    parent[2:first_sp] = 1
    parent[first_sp:first_st] = 2 + np.arange(n_sp) // SPECIES
    parent[first_st:] = first_sp + np.arange(genomes) // STRAINS
    return parent, np.arange(first_st, first_st + genomes, dtype=np.uint32)


def _letters(alphabet):
    return torch.tensor(list(alphabet), dtype=torch.uint8, device="cuda")


def _random_bases(shape, g):
    return _letters(b"ACGT")[torch.randint(0, 4, shape, generator=g, device="cuda", dtype=torch.uint8).int()]


def _spots(n, rate, g):
    """Positions in [0, n), one in each stretch of 1 / rate (so no two alike)."""
    step = max(1, int(1 / rate))
    at = torch.arange(n // step, device="cuda") * step
    return at + torch.randint(0, step, at.shape, generator=g, device="cuda")


def _substitute(seq, rate, g):
    """Random bases at the given rate."""
    flat = seq.view(-1)
    at = _spots(flat.numel(), rate, g)
    flat[at] = _random_bases(at.shape, g)
    return seq


def _genomes(count, length, related, g):
    """count rows of length bases: independent, or strains 1% from their
    species, species 4% from their genus."""
    if not related:
        return _random_bases((count, length), g)
    n_sp = -(-count // STRAINS)
    genus = _random_bases((-(-n_sp // SPECIES), length), g)
    species = _substitute(genus.repeat_interleave(SPECIES, 0)[:n_sp].contiguous(), 0.04, g)
    return _substitute(species.repeat_interleave(STRAINS, 0)[:count].contiguous(), 0.01, g)


def _bits(n):
    return max(1, (n - 1).bit_length())


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _minimizers(db, rows):
    """Minimizer of every k-mer of the rows (int64, rows x k-mers)."""
    n, ln = rows.shape
    off = torch.arange(n + 1, dtype=torch.int64, device="cuda") * ln
    mins = torch.empty(n * ln, dtype=torch.int64, device="cuda")
    amb = torch.empty(n * ln, dtype=torch.uint8, device="cuda")
    db.scan(rows.data_ptr(), off.data_ptr(), n, mins.data_ptr(), amb.data_ptr(), _stream())
    return mins.view(n, ln)[:, :ln - K + 1]


def _table(cells, related, wide, g):
    """A database of `cells` cells at load 0.7 and the genomes in it."""
    source = min(200_000_000, int(cells * LOAD * 2.2))
    count = max(16, min(8192, source // 50_000)) // 16 * 16
    rows = _genomes(count, max(400, source // count), related, g)
    parent, taxa = _taxonomy(count)
    vb = _bits(len(parent))
    db = k2g.Database.create(_options(), cells, (40 if wide else 32) - vb, vb, parent)
    step = max(1, 100_000_000 // rows.shape[1])
    tx = torch.from_numpy(taxa.view(np.int32)).cuda()
    for r in range(0, count, step):
        keys = _minimizers(db, rows[r:r + step])
        new = torch.ones_like(keys, dtype=torch.bool)
        new[:, 1:] = keys[:, 1:] != keys[:, :-1]
        owner = tx[r:r + step, None].expand_as(keys)[new].contiguous()
        keys = keys[new].contiguous()
        db.build_insert(keys.data_ptr(), owner.data_ptr(), keys.numel(), True, _stream())
    del keys, owner, new
    left = int(cells * LOAD) - db.info().size
    while left > 0:
        n = min(left, 1 << 28)
        keys = torch.randint(0, 1 << 62, (n,), generator=g, device="cuda", dtype=torch.int64)
        owner = torch.randint(1, len(parent), (n,), generator=g, device="cuda", dtype=torch.int32)
        db.build_insert(keys.data_ptr(), owner.data_ptr(), n, True, _stream())
        left -= n
    return db, rows


def _reads(rows, lens, g, hit_share=0.75, subs=0.01, n_rate=0.0, pairs=False):
    """Reads of the given lengths (numpy) from the rows, one after another;
    with pairs, sequences 2i and 2i + 1 face each other some 300 bases apart.
    Returns (bases with 16 bytes of padding, offsets)."""
    count, ln = rows.shape
    n = len(lens)
    off = np.zeros(n + 1, np.int64)
    np.cumsum(lens, out=off[1:])
    total = int(off[-1])
    out = torch.zeros(total + 16, dtype=torch.uint8, device="cuda")
    d_off = torch.from_numpy(off).cuda()
    d_len = d_off[1:] - d_off[:-1]
    frags = n // 2 if pairs else n
    row = torch.randint(0, count, (frags,), generator=g, device="cuda")
    span = torch.minimum(d_len.max() * (3 if pairs else 1), torch.tensor(ln, device="cuda"))
    at = (torch.rand(frags, generator=g, device="cuda", dtype=torch.float64) * (ln - span + 1)).long()
    hit = torch.rand(frags, generator=g, device="cuda") < hit_share
    if pairs:
        row, hit = row.repeat_interleave(2), hit.repeat_interleave(2)
        second = torch.arange(n, device="cuda") % 2 == 1
        gap = torch.randint(0, 200, (frags,), generator=g, device="cuda").repeat_interleave(2)
        at = at.repeat_interleave(2) + torch.where(second, gap, 0)
        at = torch.minimum(at, ln - d_len)
    flat = rows.reshape(-1)
    comp = torch.zeros(256, dtype=torch.uint8, device="cuda")
    comp[_letters(b"ACGT").long()] = _letters(b"TGCA")
    step = 1 + int(60_000_000 // max(1, lens.max()))
    for a in range(0, n, step):
        z = min(n, a + step)
        m = int(off[z] - off[a])
        ids = torch.repeat_interleave(torch.arange(a, z, device="cuda"), d_len[a:z], output_size=m)
        within = torch.arange(m, device="cuda") + int(off[a]) - d_off[ids]
        src = flat[row[ids] * ln + at[ids] + within]
        if pairs:
            back = flat[row[ids] * ln + at[ids] + d_len[ids] - 1 - within]
            src = torch.where(second[ids], comp[back.long()], src)
        out[int(off[a]):int(off[z])] = torch.where(hit[ids], src, _random_bases((m,), g))
    body = out[:total]
    _substitute(body, subs, g)
    if n_rate:
        body[_spots(total, n_rate, g)] = ord("N")
    return out, d_off, off


def _lengths(case, seed, n):
    r = np.random.default_rng(seed)
    lo, hi = case["len_min"], case["len_max"]
    return np.full(n, hi, np.int64) if lo == hi else r.integers(lo, hi + 1, n)


def _device_call(db, bases, quals, d_off, n_frags, max_len, total, params, runs_cap):
    """The buffers and argument blocks of one k2g_classify call."""
    nodes = int(db.info().node_count)
    zero = torch.zeros(nodes + 1, dtype=torch.int64, device="cuda")   # taxon reads, status word
    z = lambda m, t: torch.zeros(max(int(m), 1), dtype=t, device="cuda")  # noqa: E731
    out = {"call": z(n_frags, torch.int32), "hit_groups": z(n_frags, torch.int32),
           "hitlist_off": z(n_frags, torch.int64), "hitlist_len": z(n_frags, torch.int32),
           "runs": z(runs_cap, torch.int64), "taxon_reads": zero[:nodes]}
    reads = k2g.Reads(bases.data_ptr(), quals.data_ptr() if quals is not None else None,
                      d_off.data_ptr(), n_frags, max_len, total, None, 0)
    res = k2g.Results(out["call"].data_ptr(), out["hit_groups"].data_ptr(),
                      out["hitlist_off"].data_ptr(), out["hitlist_len"].data_ptr(),
                      out["runs"].data_ptr(), runs_cap, zero.data_ptr(), None, None, None, 0, None,
                      zero[nodes:].data_ptr())
    return {"kind": "device", "db": db, "zero": zero, "out": out, "reads": reads, "res": res,
            "params": params, "keep": (bases, quals, d_off)}


def _prepare_device(case, seed):
    g = _gen(seed)
    db, rows = _table(case["cells"], case["related"], case["wide"], g)
    n = case["reads"]
    per = 2 if case["paired"] else 1
    lens = _lengths(case, seed, n * per)
    bases, d_off, off = _reads(rows, lens, g, n_rate=case["n_rate"], pairs=case["paired"])
    del rows
    total = int(off[-1])
    quals = None
    if case["quality"]:
        quals = (torch.randint(0, 40, (total + 16,), generator=g, device="cuda", dtype=torch.uint8)
                 .clamp_(min=8) + 33).contiguous()
        quals[torch.rand(total + 16, generator=g, device="cuda") < 0.9] = 33 + 37
    params = k2g.ClassifyParams(case["confidence"], 2, int(case["quick"]), int(case["paired"]),
                                case["quality"])
    return _device_call(db, bases, quals, d_off, n, int(lens.max()), total, params,
                        n * (per * case["len_max"] + 2) + 8)


def _pinned(t):
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    p.copy_(t)
    return p


def _prepare_host(case, seed):
    g = _gen(seed)
    db, rows = _table(case["cells"], case["related"], False, g)
    r = np.random.default_rng(seed)
    n, nl = case["reads"], case.get("long_reads", 0)
    sigma = 0.8
    longest = min(50_000, rows.shape[1])
    long_lens = np.clip(r.lognormal(math.log(5000) - sigma * sigma / 2, sigma, nl), 150,
                        longest).astype(np.int64)
    lens = np.concatenate([long_lens, np.full(n, case["length"], np.int64)])
    r.shuffle(lens)
    n += nl
    bases, d_off, off = _reads(rows, lens, g, subs=0.04 if nl else 0.01)
    del rows
    runs_cap = case["reads"] * (case["length"] // 2 + 8) + nl * 4000
    s = {"kind": case["kind"], "db": db, "n": n, "bases": _pinned(bases), "off": _pinned(d_off),
         "params": k2g.ClassifyParams(case["confidence"], 2, 0, 0, 0), "runs_cap": runs_cap,
         "nodes": int(db.info().node_count)}
    for name in ("call", "hit_groups", "hitlist_len"):
        s[name] = torch.zeros(n, dtype=torch.int32, pin_memory=True)
    s["runs"] = torch.zeros(runs_cap, dtype=torch.int64, pin_memory=True)
    if case["kind"] == "counters":
        s["blocks"] = np.ascontiguousarray((off[:-1] // BLOCK_BASES).astype(np.uint32))
    return s


def _fastq(bases, n, length):
    """Fixed-width records "@r<10 digits>", read, "+", quality 'I'."""
    w = 12 + 1 + length + 3 + length + 1
    rec = torch.empty((n, w), dtype=torch.uint8, device="cuda")
    rec[:, 0], rec[:, 1] = ord("@"), ord("r")
    ids = torch.arange(n, device="cuda")
    for d in range(10):
        rec[:, 2 + d] = (ord("0") + (ids // 10 ** (9 - d)) % 10).to(torch.uint8)
    rec[:, 12] = ord("\n")
    rec[:, 13:13 + length] = bases[:n * length].view(n, length)
    rec[:, 13 + length] = ord("\n")
    rec[:, 14 + length] = ord("+")
    rec[:, 15 + length] = ord("\n")
    rec[:, 16 + length:16 + 2 * length] = ord("I")
    rec[:, 16 + 2 * length] = ord("\n")
    return rec.view(-1)


def _prepare_text(case, seed):
    g = _gen(seed)
    db, rows = _table(case["cells"], case["related"], False, g)
    n, length = case["reads"], case["length"]
    bases, _, _ = _reads(rows, np.full(n, length, np.int64), g)
    nodes = int(db.info().node_count)
    db.set_names(np.arange(nodes, dtype=np.uint64), [b"t%d" % i for i in range(nodes)])
    text = _pinned(_fastq(bases, n, length))
    params = k2g.ClassifyParams(case["confidence"], 2, 0, 0, 0)
    return {"kind": "text", "db": db, "text": text, "chunk": case["chunk"], "nodes": nodes,
            "reader": k2g.TextReader(db, params, chunk_cap=case["chunk"]),
            "out": torch.zeros(n * (length + 60), dtype=torch.uint8, pin_memory=True)}


AMINO = b"ACDEFGHIKLMNPQRSTVWY"
CODON = {"A": b"GCT", "C": b"TGC", "D": b"GAC", "E": b"GAA", "F": b"TTC", "G": b"GGA", "H": b"CAC",
         "I": b"ATC", "K": b"AAG", "L": b"CTG", "M": b"ATG", "N": b"AAC", "P": b"CCG", "Q": b"CAG",
         "R": b"CGT", "S": b"TCC", "T": b"ACG", "V": b"GTC", "W": b"TGG", "Y": b"TAC"}


def _prepare_translated(case, seed):
    g = _gen(seed)
    count = 64
    ln = case["residues"] // count
    which = torch.randint(0, len(AMINO), (count, ln), generator=g, device="cuda")
    parent, taxa = _taxonomy(count)
    vb = _bits(len(parent))
    db = k2g.Database.create(_options(True), int(case["residues"] / 1.6) | 1, 32 - vb, vb, parent)
    db.build_sequences(_letters(AMINO)[which].reshape(-1).cpu().numpy(),
                       np.arange(count + 1, dtype=np.uint64) * ln, taxa)
    codons = torch.tensor([list(CODON[chr(a)]) for a in AMINO], dtype=torch.uint8, device="cuda")
    dna = codons[which].reshape(count, 3 * ln)
    comp = torch.zeros(256, dtype=torch.uint8, device="cuda")
    comp[_letters(b"ACGT").long()] = _letters(b"TGCA")
    both = torch.cat([dna, comp[dna.long()].flip(1)])   # reads of either strand
    n, length = case["reads"], case["length"]
    bases, d_off, off = _reads(both, np.full(n, length, np.int64), g, hit_share=0.9)
    total = int(off[-1])
    return _device_call(db, bases, None, d_off, n, length, total,
                        k2g.ClassifyParams(0.0, 2, 0, 0, 0), 2 * total + 32 * n + 16)


def _prepare_lookup(case, seed):
    g = _gen(seed)
    db, rows = _table(case["cells"], False, False, g)
    n = case["keys"]
    mins = _minimizers(db, rows[:max(1, min(len(rows), 64_000_000 // rows.shape[1]))]).reshape(-1)
    keys = mins[torch.randint(0, mins.numel(), (n,), generator=g, device="cuda")]
    rnd = torch.randint(0, 1 << 62, (n,), generator=g, device="cuda", dtype=torch.int64)
    keys = torch.where(torch.rand(n, generator=g, device="cuda") < 0.7, keys, rnd)
    return {"kind": "lookup", "db": db, "keys": keys,
            "vals": torch.zeros(n, dtype=torch.int32, device="cuda")}


def _prepare_build(case, seed):
    g = _gen(seed)
    count = case["genomes"]
    ln = case["bases"] // count
    rows = _genomes(count, ln, True, g)
    parent, taxa = _taxonomy(count)
    return {"kind": "build", "bases": _pinned(rows.view(-1)).numpy(), "taxa": taxa, "parent": parent,
            "off": np.arange(count + 1, dtype=np.uint64) * ln, "cells": case["cells"]}


def prepare(case, seed):
    make = {"device": _prepare_device, "host": _prepare_host, "counters": _prepare_host,
            "text": _prepare_text, "translated": _prepare_translated, "lookup": _prepare_lookup,
            "build": _prepare_build}
    return make[case["kind"]](case, seed)


# ---- one pass ---------------------------------------------------------------

def _run_device(s):
    s["zero"].zero_()
    s["db"].classify(s["reads"], s["params"], s["res"], mode=k2g.MODE_PIPELINED, stream=_stream())
    return s["out"]


def _run_host(s):
    runs = C.c_uint64(s["runs_cap"])
    args = (s["call"].data_ptr(), s["hit_groups"].data_ptr(), s["hitlist_len"].data_ptr(),
            s["runs"].data_ptr(), C.byref(runs))
    taxon_reads = np.zeros(s["nodes"], np.uint64)
    counters = None
    if s["kind"] == "counters":
        counters = k2g.Counters(s["db"])
        k2g.check(k2g.lib().k2g_classify_host_blocks(
            s["db"].h, s["bases"].data_ptr(), None, s["off"].data_ptr(), s["n"],
            s["blocks"].ctypes.data, counters.h, C.byref(s["params"]), *args,
            taxon_reads.ctypes.data))
    else:
        k2g.check(k2g.lib().k2g_classify_host(
            s["db"].h, s["bases"].data_ptr(), None, s["off"].data_ptr(), s["n"],
            C.byref(s["params"]), *args, taxon_reads.ctypes.data))
    out = {"call": s["call"], "hit_groups": s["hit_groups"], "hitlist_len": s["hitlist_len"],
           "runs": s["runs"], "n_runs": int(runs.value), "taxon_reads": taxon_reads.view(np.int64)}
    if counters is not None:
        kmers, clade_kmers, clade_distinct = counters.finish(_stream())
        counters.close()
        out.update(kmers=kmers.view(np.int64), clade_kmers=clade_kmers.view(np.int64),
                   clade_distinct=clade_distinct.view(np.int64))
    return out


def _run_text(s):
    lib, h = k2g.lib(), s["reader"].h
    s["reader"].reset()
    base_in, base_out, total = s["text"].data_ptr(), s["out"].data_ptr(), s["text"].numel()
    pos = got = frags = classified = 0
    k2g.check(lib.k2g_text_prefetch(h, base_in, min(s["chunk"], total)))
    while pos < total:
        n = min(s["chunk"], total - pos)
        if pos + n < total:   # the next chunk's copy runs beside this chunk's work
            k2g.check(lib.k2g_text_prefetch(h, base_in + pos + n, min(s["chunk"], total - pos - n)))
        res = k2g.TextResult()
        k2g.check(lib.k2g_text_classify(h, base_in + pos, n, int(pos + n >= total), None, C.byref(res)))
        if res.handoff or got + res.text_len > s["out"].numel():
            raise RuntimeError("the input left the strict form or its lines the buffer")
        k2g.check(lib.k2g_text_fetch_async(h, base_out + got, res.text_len))
        got += res.text_len
        frags += res.fragments
        classified += res.classified
        pos += n
    k2g.check(lib.k2g_text_wait(h))
    taxon_reads = np.zeros(s["nodes"], np.uint64)
    s["reader"].taxon_reads(taxon_reads)
    return {"lines": s["out"], "bytes": got, "fragments": frags, "classified": classified,
            "taxon_reads": taxon_reads.view(np.int64)}


def _run_lookup(s):
    s["db"].lookup(s["keys"].data_ptr(), s["vals"].data_ptr(), s["keys"].numel(), _stream())
    return s["vals"]


class _DeviceWords:
    """The table's 32-bit cells as a CUDA array."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": "<i4",
                                         "version": 3}


def _run_build(s):
    vb = _bits(len(s["parent"]))
    db = k2g.Database.create(_options(), s["cells"], 32 - vb, vb, s["parent"])
    pairs = db.build_sequences(s["bases"], s["off"], s["taxa"])
    info = db.info()
    cells = torch.as_tensor(_DeviceWords(info.d_cells, s["cells"]), device="cuda").clone()
    torch.cuda.current_stream().synchronize()   # the copy ends before the table is given back
    db.close()
    return {"cells": cells, "size": int(info.size), "pairs": pairs}


def run(state):
    go = {"device": _run_device, "host": _run_host, "counters": _run_host, "text": _run_text,
          "lookup": _run_lookup, "build": _run_build}
    return go[state["kind"]](state)


# ---- what a pass cannot do without -------------------------------------------

def _lookups(length):
    """Distinct minimizers of a read: about one in three of its k-mers."""
    return max(0.0, (length - K + 1) / 3)


def work(case):
    kind = case["kind"]
    if kind == "lookup":
        return {"bytes": case["keys"] * (8 + 4 + min(32, 4 * case["cells"] / case["keys"])), "flops": 0.0}
    if kind == "build":
        return {"bytes": case["bases"] + 4 * case["cells"], "flops": 0.0}
    if kind == "translated":
        # six frames of a third of the bases each, a new minimizer every second residue
        frame = case["length"] / 3 - PROTEIN_K + 1
        sectors = case["reads"] * max(0.0, 6 * frame / 2.5)
        table = 4 * case["residues"] / 1.6
        return {"bytes": case["reads"] * (case["length"] + 8 + 20 + 8 * 12) + min(32 * sectors, table),
                "flops": 0.0}
    cell = 8 if case.get("wide") else 4
    if kind == "device":
        per = 2 if case["paired"] else 1
        mean = (case["len_min"] + case["len_max"]) / 2
        reads = case["reads"] * (per * (mean * (2 if case["quality"] else 1) + 8) + 20 + 8 * 5)
        sectors = case["reads"] * per * _lookups(mean)
        return {"bytes": reads + min(32 * sectors, cell * case["cells"]), "flops": 0.0}
    n, nl = case["reads"], case.get("long_reads", 0)
    bases = n * case["length"] + nl * 5000
    sectors = n * _lookups(case["length"]) + nl * _lookups(5000)
    moved = bases + (n + nl) * (8 + 20) + 8 * (5 * n + 600 * nl)
    if kind == "text":
        moved = n * (2 * case["length"] + 17) + n * 60
    return {"bytes": moved + min(32 * sectors, cell * case["cells"]), "flops": 0.0}


def exact(case, seed):
    """Every output is a whole number or a byte: there is no rounding to compare."""
    return None
