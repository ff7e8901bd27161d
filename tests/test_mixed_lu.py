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
    assert _complex_error(got, ref, omegas) <= 1e-5


def _complex_error(got, ref, omegas):
    """The largest error of A - i B / omega and of X against their entries' scales."""
    z, r = (np.asarray(q["A"]) - 1j * np.asarray(q["B"]) / omegas[:, None, None] for q in (got, ref))
    pairs = [(z, r)] + ([(np.asarray(got["X"]), np.asarray(ref["X"]))] if np.asarray(ref["X"]).size else [])
    return max(float((np.abs(a - b) / np.maximum(np.abs(b).max(axis=0, keepdims=True), 1e-3 * np.abs(b).max())).max())
               for a, b in pairs)


@pytest.mark.gpu
@pytest.mark.parametrize("freqs,headings", [(1, 0), (2, 1), (3, 3), (64, 4), (96, 6), (96, 9), (5, 13), (150, 14), (40, 26)])
def test_sweep_columns(freqs, headings):
    """The triangular sweeps' column pairs (odd counts, a short last group) and group sizes, from one system, whose
    columns are spread over the SMs, to many, which keep them together: 3 blocks of 128 rows, 380 panels."""
    from hydrobem_b200 import native as nv

    v = meshes.cylinder(1.0, 0.5, 20, 9, 10)
    omegas = np.sqrt(np.linspace(0.4, 1.2, freqs) * meshes.GRAVITY)
    heads = 7.0 * np.arange(headings)
    ref = nv.solve(v, omegas, heads, depth=math.inf, precision=nv.HBG_FP64)
    got = nv.solve(v, omegas, heads, depth=math.inf, precision=nv.HBG_MIXED)
    assert nv.last_fallback_count() == 0
    hist = nv.last_ir_history()
    assert all(b < 5e-3 * a for a, b in zip(hist, hist[1:])), hist
    assert _complex_error(got, ref, omegas) <= 1e-5
