"""The first mixed solve on fresh buffers, and one on buffers that another problem has filled, are the later ones to the bit:
every sum has a fixed order, so an entry that is read before it is written shows."""
from __future__ import annotations

import math

import numpy as np
import pytest

from hydrobem_b200 import meshes


@pytest.mark.gpu
@pytest.mark.parametrize("freqs,headings,depth", [(1, 0, math.inf), (12, 2, math.inf), (12, 12, 4.0), (5, 26, math.inf)])
def test_first_solve(freqs, headings, depth):
    from hydrobem_b200 import native as nv

    v = meshes.cylinder(1.0, 0.5, 40, 14, 14)  # 1120 panels
    omegas = np.sqrt(np.linspace(0.4, 1.2, freqs) * meshes.GRAVITY)
    heads = 7.0 * np.arange(headings)
    solve = lambda: nv.solve(v, omegas, heads, depth=depth, precision=nv.HBG_MIXED)  # noqa: E731
    nv.lib().hbg_release_workspace()
    runs = [solve(), solve()]
    nv.solve(meshes.cylinder(2.0, 0.7, 48, 16, 17), 0.8 * omegas, heads + 3.0, depth=5.0, precision=nv.HBG_MIXED)
    runs.append(solve())
    for q in runs[1:]:
        for key in ("A", "B", "X", "HK"):
            assert np.array_equal(np.asarray(q[key]), np.asarray(runs[0][key])), key
