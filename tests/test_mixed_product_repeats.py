"""The mixed form's FP64 product against numpy, and hundreds of times over: every sum has a fixed order, so results that
are not the first's to the bit show a stage of the product's ring that was refilled while it was still being read."""
from __future__ import annotations

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n,batch,nrhs,repeats", [(16, 1, 1, 5), (127, 3, 6, 50), (640, 40, 7, 400), (1050, 24, 8, 400),
                                                  (1050, 24, 10, 200), (1280, 24, 13, 200), (900, 24, 19, 200), (700, 24, 24, 200),
                                                  (700, 24, 27, 200), (2300, 4, 32, 100)])
def test_product(n, batch, nrhs, repeats):
    from hydrobem_b200 import native as nv

    rng = np.random.default_rng(n + nrhs)
    M = (rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))).astype(np.complex64)
    x = rng.standard_normal((batch, nrhs, n)) + 1j * rng.standard_normal((batch, nrhs, n))
    y, differ = nv.debug_cgemv(M, x, repeats)
    assert differ == 0
    # a sum of 2 n products a component, in any order: at most 2 n eps of the sum of their moduli (2 |M| |x| an entry)
    ref = np.einsum("bkn,bcn->bck", M.astype(np.complex128), x, optimize=True)
    scale = np.einsum("bkn,bcn->bck", np.abs(M).astype(np.float64), np.abs(x), optimize=True)
    assert (np.abs(y - ref) <= 8.0 * n * 2.0 ** -53 * scale).all()
