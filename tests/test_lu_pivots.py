"""The FP64 form's pivots: the largest modulus of the column to the last bit of |a|^2, the first row on a tie."""
from __future__ import annotations

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n,batch", [(64, 3), (300, 2), (1200, 2), (2500, 1), (4400, 1), (270, 230)])
def test_near_ties(n, batch):
    """Columns i and i + n / 2 meet rows i and i + n / 2 alone, so that the interchange of column i is known: its two
    candidates differ by 2^-36, or by nothing."""
    from hydrobem_b200 import native as nv

    rng = np.random.default_rng(n)
    h = n // 2
    i = np.arange(h)
    A = np.zeros((batch, n, n), np.complex128)
    want = np.zeros((batch, n), np.int32)
    for f in range(batch):
        d = rng.choice([-1, 0, 1], h)
        first, second = 1.25 * (1.0 + 2.0 ** -36 * (d < 0)), 1.25 * (1.0 + 2.0 ** -36 * (d > 0))
        A[f, i, i] = first * rng.choice([1, -1, 1j, -1j], h)
        A[f, i + h, i] = second * rng.choice([1, -1, 1j, -1j], h)
        A[f, i, i + h] = 1.0
        want[f] = np.arange(n)
        want[f, i] = np.where(d > 0, i + h, i)
    assert np.array_equal(nv.debug_lu_pivots(A), want)
