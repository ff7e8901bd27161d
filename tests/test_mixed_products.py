"""The mixed form's matrix products with all right-hand sides (b = S u, r = b - A x, r - A d): every count of column tiles
(6 to 32 right-hand sides, odd and full), 1120 panels (a chunk of 1024 columns and a short one, a ragged last tile of rows).

The solution is compared with the FP64 form's at the repository's bound of 1e-5 of each entry's scale, and repeated
solves are the same to the bit: every sum has a fixed order, so a product that read a tile before its load or after its
release shows."""
from __future__ import annotations

import math

import numpy as np
import pytest

from hydrobem_b200 import meshes


@pytest.mark.gpu
@pytest.mark.parametrize("headings", [0, 2, 5, 9, 12, 17, 21, 26])
def test_columns_and_repeats(headings):
    from hydrobem_b200 import native as nv

    v = meshes.cylinder(1.0, 0.5, 40, 14, 14)
    omegas = np.sqrt(np.linspace(0.4, 1.2, 12) * meshes.GRAVITY)
    heads = 7.0 * np.arange(headings)
    ref = nv.solve(v, omegas, heads, depth=math.inf, precision=nv.HBG_FP64)
    runs = [nv.solve(v, omegas, heads, depth=math.inf, precision=nv.HBG_MIXED) for _ in range(6)]
    assert nv.last_fallback_count() == 0
    z, r = (np.asarray(q["A"]) - 1j * np.asarray(q["B"]) / omegas[:, None, None] for q in (runs[-1], ref))
    pairs = [(z, r)] + ([(np.asarray(runs[-1]["X"]), np.asarray(ref["X"]))] if headings else [])
    for a, b in pairs:
        scale = np.maximum(np.abs(b).max(axis=0, keepdims=True), 1e-3 * np.abs(b).max())
        assert float((np.abs(a - b) / scale).max()) <= 1e-5
    for q in runs[2:]:
        for key in ("A", "B", "X"):
            assert np.array_equal(np.asarray(q[key]), np.asarray(runs[1][key])), key
