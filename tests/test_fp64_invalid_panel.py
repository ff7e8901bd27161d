"""An invalid panel ends the FP64 form's solve before its first factorization."""
from __future__ import annotations

import math

import numpy as np
import pytest

from hydrobem_b200 import meshes


@pytest.mark.gpu
@pytest.mark.parametrize("max_batch", [0, 1])
@pytest.mark.parametrize("concurrency", [1, 2])
def test_invalid_panel_before_the_factorization(max_batch, concurrency):
    from hydrobem_b200 import native as nv

    v = meshes.cylinder(1.0, 0.5, 32, 8, 8)  # 512 panels
    bad = v.copy()
    bad[300] = bad[300, 0]  # no area
    omegas = np.sqrt(np.array([0.3, 0.7, 1.1]) * meshes.GRAVITY)
    opt = dict(depth=math.inf, precision=nv.HBG_FP64, max_batch=max_batch, concurrency=concurrency)
    with pytest.raises(nv.HydroBEMError, match="invalid panel 301 "):
        nv.solve_batch([nv.Body(bad, omegas, [20.0]) for _ in range(concurrency)], **opt)
    # geometry, hydrostatics, statics, assembly, boundary and right-hand sides: the LU of 512 panels alone is 40 launches
    assert nv.last_launch_count() <= 12 * concurrency
    assert np.isfinite(nv.solve(v, omegas, [20.0], **opt)["A"]).all()  # and the next solve is a solve
