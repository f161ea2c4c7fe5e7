"""The one-subtraction modulo of the table lookups (k2g_device.cuh), restated:
q = floor(n * floor((2^64 - 1) / d) / 2^64) is n // d or one less."""
import numpy as np
import pytest


@pytest.mark.parametrize("d", [1, 2, 3, 7, 8, 1000, 5003, 2**31 - 1, 2**32, 2**32 + 1, 10_000_000_000,
                               14_285_714_285, 2**40 + 12345, 2**63 - 25, 2**63])
def test_one_subtraction_is_enough(d):
    rng = np.random.default_rng(d % 997)
    inv = (2**64 - 1) // d
    top = (2**64 - 1) // d * d
    ns = [0, 1, d - 1, d, d + 1, 2 * d - 1, 2**64 - 1, 2**64 - d, top, top - 1, top - d, top - d - 1]
    ns += [int(x) for x in rng.integers(0, 2**64 - 1, 400, dtype=np.uint64)]
    for n in ns:
        n %= 2**64
        r = n - ((n * inv) >> 64) * d
        assert 0 <= r < 2 * d
        assert (r - d if r >= d else r) == n % d
