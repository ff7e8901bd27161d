"""The FP64 form's LU at the edges of its strips: rows that fit one CTA or clusters of two to eight, 32 and 16 columns in
registers, 8 in global memory, remainders of all, on random matrices (nearly every column swaps rows)."""
from __future__ import annotations

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n,batch", [(2, 5), (33, 3), (255, 2), (257, 9), (511, 2), (1030, 2), (2049, 1), (2300, 2), (4100, 1)])
def test_residual(n, batch):
    from hydrobem_b200 import native as nv

    rng = np.random.default_rng(n)
    A = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    B = rng.standard_normal((batch, n, 3)) + 1j * rng.standard_normal((batch, n, 3))
    X = nv.debug_lu_f64(A, B)
    for a, b, x in zip(A, B, X):
        # backward error of a pivoted LU: a small multiple of n eps |A| |X| (the growth of random matrices is mild)
        assert np.abs(a @ x - b).max() <= 1e-15 * n * np.abs(a).max() * np.abs(x).max()


@pytest.mark.gpu
def test_pivot_order_of_equal_moduli():
    """The first row of the largest modulus is taken: a matrix whose columns tie everywhere."""
    from hydrobem_b200 import native as nv

    n = 300
    i = np.arange(n)
    A = np.exp(2j * np.pi * np.outer(i, i) / n)[None]  # the discrete Fourier matrix: all moduli one
    B = np.eye(n, 2)[None].astype(np.complex128)
    X = nv.debug_lu_f64(A, B)
    assert np.abs(X[0] - A[0].conj()[:, :2] / n).max() <= 1e-13


@pytest.mark.gpu
def test_residual_of_many_matrices():
    """More matrices than the strips' clusters may take SMs for: strips of 8 in global memory, then of 32 columns once the
    rows fit one CTA."""
    from hydrobem_b200 import native as nv

    n, batch = 270, 230
    rng = np.random.default_rng(n)
    A = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    B = rng.standard_normal((batch, n, 3)) + 1j * rng.standard_normal((batch, n, 3))
    X = nv.debug_lu_f64(A, B)
    assert np.abs(A @ X - B).max() <= 1e-15 * n * np.abs(A).max() * np.abs(X).max()
