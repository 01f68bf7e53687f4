"""The kernels' quotients by multiplication (reciprocal in csrc/dmmv_slice.cuh): exact wherever the host hands one out."""
import numpy as np
import pytest

from helpers import run_cpp


def reciprocal(d, limit):
    return 2 ** 32 // d + 1 if d > 1 and limit * d < 2 ** 32 else 0


@pytest.mark.parametrize("d", [1, 2, 3, 5, 6, 32, 147, 180, 205, 4095, 4096, 16384, 65535])
def test_quotient_is_exact(d):
    for limit in (1, d, 9 * d, 32 * d, 65536, 2 ** 32 // d, (2 ** 32 - 1) // d):
        mul = reciprocal(d, limit)
        if not mul:
            assert d == 1 or limit * d >= 2 ** 32
            continue
        step = max(1, limit // 4096)
        n = np.unique(np.concatenate([np.arange(0, limit, step), np.arange(0, limit, d)[:100000], np.arange(d - 1, limit, d)[-100000:],
                                      [limit - 1]])).astype(np.uint64)
        assert np.array_equal((n * np.uint64(mul)) >> np.uint64(32), n // np.uint64(d))


def test_the_kernels_own():
    """reciprocal, quotient and the limits in slice_plan, compiled for the host from the kernels' header."""
    run_cpp("test_reciprocal")
