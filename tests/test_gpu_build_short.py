"""k2g_build_sequences on short sequences, around the candidates a block from
which blocks are sorted each by itself: the same lists as made by hand."""
import numpy as np
import pytest

import test_gpu_build_blocks as blocks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [36, 60, 100, 108, 112, 150])      # (108: 24 candidates on average)
def test_short_sequences(length, monkeypatch):
    def library(kind, rng):
        acgt = np.frombuffer(b"ACGT", np.uint8)
        return [acgt[rng.integers(0, 4, length - i % 2)] for i in range(400)]

    monkeypatch.setattr(blocks, "library", library)
    blocks.test_list_equals_scan_by_hand("short", 16384, 1024)
