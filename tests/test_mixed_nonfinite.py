"""A correction of the refinement that is not finite counts as one that does not contract: the frequency goes to the FP64
form instead of passing for converged."""
from __future__ import annotations

import math

import numpy as np
import pytest

from hydrobem_b200 import meshes


@pytest.mark.gpu
def test_right_hand_sides_beyond_fp32():
    """Rotations about a centre 1e39 away: right-hand sides (and residuals) that FP32 cannot hold, FP64 can."""
    from hydrobem_b200 import native as nv

    v = meshes.cylinder(1.0, 0.5, 16, 8, 7)
    omegas = np.sqrt(np.array([0.3, 1.1]) * meshes.GRAVITY)
    kw = dict(headings_deg=[20.0], rotation_centers=[[1e39, 0.0, 0.0]], depth=math.inf)
    ref = nv.solve(v, omegas, precision=nv.HBG_FP64, **kw)
    assert np.isfinite(ref["A"]).all()
    got = nv.solve(v, omegas, precision=nv.HBG_MIXED, **kw)
    assert nv.last_fallback_count() == 2
    for q in ("A", "B", "X"):
        a, b = np.asarray(got[q]), np.asarray(ref[q])
        assert np.abs(a - b).max(initial=0.0, where=np.abs(b) < 1e30) <= 1e-12 * np.abs(b[np.abs(b) < 1e30]).max()
        assert (np.abs(a - b) <= 1e-12 * np.abs(b).max()).all()
