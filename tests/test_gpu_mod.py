"""The modulo of the table lookups as the kernels compute it (mod_once, and
fast_mod beside it) with the library's constants, at divisors from 1 to 2^63
and dividends at the multiples of each."""
import os
import subprocess

import numpy as np
import pytest

from kraken2_gb300 import build as kb

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
DIVISORS = [1, 2, 3, 7, 8, 1000, 5003, 1_000_003, 2**31 - 1, 2**31, 2**32 - 1, 2**32, 2**32 + 1, 10_000_000_000,
            14_285_714_285, 2**40 - 1, 2**40, 2**40 + 12345, 2**62 + 3, 2**63 - 25, 2**63 - 1, 2**63]


def test_remainders_equal_those_of_integers(tmp_path):
    kb.build()
    exe = str(tmp_path / "mod_check")
    subprocess.run([kb.nvcc(), *kb.ARCH, *kb.COMMON, os.path.join(HERE, "mod_check.cu"), "-L", kb.OUT, "-lk2g",
                    "-Xlinker", "-rpath=" + kb.OUT, "-o", exe], check=True)
    rng = np.random.default_rng(1)
    asked, text = [], b""
    for d in DIVISORS:
        top = (2**64 - 1) // d * d
        ns = [0, 1, d - 1, d, d + 1, 2 * d - 1, 2**64 - 1, 2**64 - d, top, top - 1, top - d, top - d - 1]
        ns += [q * d + r for q in (int(x) for x in rng.integers(0, (2**64 - 1) // d, 300, dtype=np.uint64, endpoint=True))
               for r in (-1, 0, 1)]
        ns += [int(x) for x in rng.integers(0, 2**64 - 1, 2000, dtype=np.uint64)]
        ns = [n % 2**64 for n in ns]
        asked.append((d, ns))
        text += np.array([len(ns), d] + ns, np.uint64).tobytes()
    out = subprocess.run([exe], input=text, stdout=subprocess.PIPE, check=True).stdout
    got = np.frombuffer(out, np.uint64).reshape(-1, 2)
    want = [n % d for d, ns in asked for n in ns]
    assert len(got) == len(want)
    assert got[:, 0].tolist() == want and got[:, 1].tolist() == want
