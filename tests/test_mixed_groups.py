"""The mixed form's LU on several stream groups of few large systems: two and three groups of two to seven systems (uneven
and single ones), from the smallest orders that take them, and the groups of eight systems beside them."""
from __future__ import annotations

import math

import numpy as np
import pytest

from hydrobem_b200 import meshes


@pytest.mark.gpu
@pytest.mark.parametrize("n_phi,n_z,n_r,freqs", [(48, 20, 20, 3), (48, 22, 23, 2), (48, 22, 23, 4), (48, 22, 23, 5), (48, 22, 23, 7),
                                                 (64, 20, 20, 8), (64, 40, 41, 3), (64, 40, 41, 5)])
def test_few_large_systems(n_phi, n_z, n_r, freqs):
    from hydrobem_b200 import native as nv

    v = meshes.cylinder(1.0, 0.5, n_phi, n_z, n_r)  # 1920, 2160, 2560, 5184 panels
    omegas = np.sqrt(np.linspace(0.3, 1.1, freqs) * meshes.GRAVITY)
    ref = nv.solve(v, omegas, [20.0], depth=math.inf, precision=nv.HBG_FP64)
    got = nv.solve(v, omegas, [20.0], depth=math.inf, precision=nv.HBG_MIXED)
    assert nv.last_fallback_count() == 0
    hist = nv.last_ir_history()  # (TF32 and FP16 factors of mild systems: a correction leaves about 1e-3, a wrong block 1e-2)
    assert all(b < 5e-3 * a for a, b in zip(hist, hist[1:])), hist
    z, r = (np.asarray(q["A"]) - 1j * np.asarray(q["B"]) / omegas[:, None, None] for q in (got, ref))
    for a, b in ((z, r), (np.asarray(got["X"]), np.asarray(ref["X"]))):  # the repository's 1e-5 of each entry's scale
        scale = np.maximum(np.abs(b).max(axis=0, keepdims=True), 1e-3 * np.abs(b).max())
        assert float((np.abs(a - b) / scale).max()) <= 1e-5
