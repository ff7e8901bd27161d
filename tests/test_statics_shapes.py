"""The statics kernels at the edges of their work split: few panels (four rows a warp) and more (32), remainders of both,
images near and far (every order of the log rule, the adaptive rule), against the oracle at 1e-10 of each plane's scale."""
from __future__ import annotations

import math

import numpy as np
import pytest

from hydrobem_b200 import meshes


@pytest.mark.gpu
@pytest.mark.parametrize("depth", [math.inf, 2.0])
@pytest.mark.parametrize("n_phi,n_z,n_r", [(3, 1, 1), (7, 3, 2), (16, 10, 13), (21, 15, 15)])
def test_statics_against_the_oracle(depth, n_phi, n_z, n_r):
    from hydrobem_b200 import native as nv
    from oracle import oracle as O

    v = meshes.cylinder(1.0, 0.3, n_phi, n_z, n_r)  # 6, 35, 368, 630 panels
    st = nv.debug_matrices(v, 1.3, depth=depth)[0]
    ref = O.statics(O.make_panels(v), None, depth)
    for q in range(4):
        assert np.abs(st[..., q] - ref[..., q]).max() <= 1e-10 * np.abs(ref[..., q]).max(), q
