"""The division by a multiplication that the GEMMs' work items are numbered with (csrc/qgemm_common.cuh, quotient): exact for every 32-bit number."""

import numpy as np
import pytest


def divide_by(d):
    return (2 ** 64 - 1) // d + 1 if d > 1 else 0


def quotient(n, by):
    return n if by == 0 else by * n >> 64


@pytest.mark.parametrize("divisors", [range(1, 300), (2 ** 16 - 1, 2 ** 16, 2 ** 16 + 1, 37888, 2 ** 31, 2 ** 32 - 1)])
def test_exact(divisors):
    rng = np.random.default_rng(1)
    for d in divisors:
        by = divide_by(d)
        assert by < 2 ** 64
        top = (2 ** 32 - 1) // d
        around = [m * d + e for m in {0, 1, 2, 3, top // 2, top - 1, top, *map(int, rng.integers(0, top + 1, 20))} for e in (-1, 0, 1)]
        for n in around + [2 ** 32 - 1] + [int(x) for x in rng.integers(0, 2 ** 32, 20)]:
            if 0 <= n < 2 ** 32:
                assert quotient(n, by) == n // d, (n, d)
