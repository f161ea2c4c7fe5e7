"""Translated search by warps against the oracle, at the lengths where codon
classes, a lane's residues, a pass and the packed window begin and end."""
import os

import numpy as np
import pytest

import kraken2_gb300 as k2g
import oracle
from gpu_util import to_dev
from test_gpu_warp import batch, check

pytestmark = pytest.mark.gpu

K, L, TOGGLE = 15, 12, 0xe37e28c4271b5a2d
AMINO = np.frombuffer(b"ACDEFGHIKLMNPQRSTVWY", np.uint8)
CODON = {"A": "GCT", "C": "TGC", "D": "GAC", "E": "GAA", "F": "TTC", "G": "GGA", "H": "CAC", "I": "ATC",
         "K": "AAG", "L": "CTG", "M": "ATG", "N": "AAC", "P": "CCG", "Q": "CAG", "R": "CGT", "S": "TCC",
         "T": "ACG", "V": "GTC", "W": "TGG", "Y": "TAC"}
# around: a codon; k residues of each class; 8 residues a lane; the packed mate
EDGES = [0, 1, 2, 3, 4, 5, 40, 43, 44, 45, 46, 47, 48, 49, 57, 58, 59, 66, 67, 68, 69, 70, 71, 72, 100, 149,
         150, 151, 152, 200, 299, 300, 301, 302, 303, 700, 1534, 1535, 1536, 1537, 1538, 1560, 3071, 3100, 5000]

_cache = {}


def database(wide, many):
    if (wide, many) in _cache:
        return _cache[wide, many]
    rng = np.random.default_rng(23)
    prot = AMINO[rng.integers(0, 20, 30_000)]
    nodes = 1500
    parent = np.zeros(nodes, np.uint64)
    parent[2:] = (rng.random(nodes - 2) * np.minimum(np.arange(1, nodes - 1), 100)).astype(np.uint64) + 1
    vb = 11
    db = k2g.Database.create(k2g.IndexOptions(K, L, 0, TOGGLE, 0, 1, 0), 40_009, (40 if wide else 32) - vb, vb,
                             parent)
    step = 18 if many else 300     # residues of one taxon
    cuts = np.arange(0, len(prot) - step, step)
    off = np.concatenate([np.stack([cuts, cuts + step + K - 1], 1).reshape(-1)])
    seqs = b"".join(bytes(prot[a:b]) for a, b in off.reshape(-1, 2))
    lens = np.diff(off.reshape(-1, 2), axis=1)[:, 0]
    so = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    db.build_sequences(seqs, so, rng.integers(1, nodes, len(lens)).astype(np.uint32))
    dna = "".join(CODON[chr(c)] for c in prot).encode()
    comp = bytes.maketrans(b"ACGT", b"TGCA")
    genome = np.frombuffer(dna + dna[::-1].translate(comp), np.uint8)
    cells, _ = db.download()
    inf = db.info()
    o = oracle.Oracle(cells, inf.capacity, inf.key_bits, inf.value_bits, parent,
                      oracle.index_opts(K, L, 0, TOGGLE, 1, 0, protein=True))
    _cache[wide, many] = (db, genome, o)
    return _cache[wide, many]


PARAMS = [dict(confidence=0.0, min_hit_groups=0), dict(confidence=0.1, min_hit_groups=2),
          dict(confidence=0.0, min_hit_groups=2, min_quality=8), dict(confidence=0.0, min_hit_groups=3, quick=True),
          dict(confidence=0.3, min_hit_groups=1, paired=True),
          dict(confidence=0.0, min_hit_groups=2, paired=True, quick=True, min_quality=5)]


@pytest.mark.parametrize("many", [False, True], ids=["stretches", "many_taxa"])
@pytest.mark.parametrize("wide", [False, True], ids=["cells32", "cells40"])
@pytest.mark.parametrize("params", PARAMS, ids=lambda p: "-".join(f"{k}{v}" for k, v in p.items()))
def test_edge_lengths_equal_the_oracle(params, wide, many):
    db, genome, o = database(wide, many)
    rng = np.random.default_rng(5)
    lens = EDGES + [int(x) for x in rng.permutation(EDGES)] + [int(x) for x in rng.integers(0, 400, 200)]
    if params.get("paired"):
        lens = lens[:len(lens) // 2 * 2]
    bases, q, off = batch(genome, lens, 8, "min_quality" in params)
    check(db, o, bases, q, off, len(lens) // (2 if params.get("paired") else 1), params)


def test_two_fragments_a_warp_equal_the_oracle():
    db, genome, o = database(False, False)
    lens = [int(x) for x in np.random.default_rng(3).integers(0, 201, 8001)]
    bases, q, off = batch(genome, lens, 9)
    check(db, o, bases, q, off, len(lens), dict(confidence=0.1, min_hit_groups=2))


def test_qualities_at_another_alignment_equal_the_oracle():
    """Qualities that do not share the bases' alignment take the general form."""
    import torch
    db, genome, o = database(False, False)
    lens = [150] * 50
    bases, q, off = batch(genome, lens, 10, True)
    b = to_dev(np.frombuffer(bases + b"\0" * 16, np.uint8))
    qd = to_dev(np.frombuffer(b"\0" * 5 + q + b"\0" * 16, np.uint8))
    d_off = to_dev(off)
    n = len(lens)
    call = torch.zeros(n, dtype=torch.int32, device="cuda")
    runs = torch.zeros(int(off[-1]) + 2 * n, dtype=torch.int64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    db.classify(k2g.Reads(b.data_ptr(), qd.data_ptr() + 5, d_off.data_ptr(), n, 150, int(off[-1]), None, 0),
                k2g.ClassifyParams(0.0, 2, 0, 0, 10),
                k2g.Results(call.data_ptr(), None, None, None, runs.data_ptr(), runs.numel(), None, None, None,
                            None, 0, None, status.data_ptr()),
                stream=torch.cuda.current_stream().cuda_stream)
    want, *_ = o.classify(bases, q, off, n, threads=os.cpu_count() or 1, confidence=0.0, min_hit_groups=2,
                          min_quality=10)
    assert int(status[0]) == 0
    assert np.array_equal(call.cpu().numpy().view(np.uint32), want.astype(np.uint32))
