"""The mixed form's LU at the sizes where its blocking can go wrong: one 128 block, a panel of two, an odd last
block (alone in a super-step, within one, after a delayed update), several super-steps, padded and full blocks.

The factors only precondition the refinement, so a wrong entry shows in its contraction: with TF32 and FP16
operands (10-bit mantissa, 2^-11 a rounding) and the mild conditioning of these systems (3-6) the first correction
leaves about 1e-3; a wrong block leaves 1e-2 and more.  The solution is compared with the FP64 form's at the
repository's bound of 1e-5 of each entry's scale."""
from __future__ import annotations

import math

import numpy as np
import pytest

from hydrobem_b200 import meshes


@pytest.mark.gpu
@pytest.mark.parametrize("n_phi,n_z,n_r", [(16, 4, 4), (16, 8, 7), (20, 9, 10), (32, 12, 8), (40, 14, 14), (48, 22, 23),
                                           (64, 20, 20)])
def test_lu_block_edges(n_phi, n_z, n_r):
    from hydrobem_b200 import native as nv

    v = meshes.cylinder(1.0, 0.5, n_phi, n_z, n_r)  # 128, 240, 380, 640, 1120, 2160, 2560 panels
    omegas = np.sqrt(np.array([0.3, 1.1]) * meshes.GRAVITY)
    ref = nv.solve(v, omegas, [20.0], depth=math.inf, precision=nv.HBG_FP64)
    got = nv.solve(v, omegas, [20.0], depth=math.inf, precision=nv.HBG_MIXED)
    assert nv.last_fallback_count() == 0
    hist = nv.last_ir_history()
    # (one 128 block is factored in FP32 alone and is done after fewer corrections)
    assert all(b < 5e-3 * a for a, b in zip(hist, hist[1:])), hist
    # the potential is solved to the rounding of the complex64 matrix, relative to its modulus: A is its real
    # part, B / omega its imaginary part (which alone may be much smaller), on one scale
    z, r = (np.asarray(q["A"]) - 1j * np.asarray(q["B"]) / omegas[:, None, None] for q in (got, ref))
    scale = np.maximum(np.abs(r).max(axis=0, keepdims=True), 1e-3 * np.abs(r).max())
    assert float((np.abs(z - r) / scale).max()) <= 1e-5
    x, r = np.asarray(got["X"]), np.asarray(ref["X"])
    scale = np.maximum(np.abs(r).max(axis=0, keepdims=True), 1e-3 * np.abs(r).max())
    assert float((np.abs(x - r) / scale).max()) <= 1e-5
