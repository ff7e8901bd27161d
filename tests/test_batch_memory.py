"""The batch size when the buffers of an earlier, larger solve hold the matrices of all frequencies but not the rest, and the
device has little memory left: a smaller batch, as with no buffers held."""
from __future__ import annotations

import numpy as np
import pytest

from hydrobem_b200 import meshes


@pytest.mark.gpu
@pytest.mark.parametrize("form,free_gb", [("mixed", 2.0), ("fp64", 0.4)])
def test_many_small_systems_after_few_large_ones(form, free_gb):
    import torch

    from hydrobem_b200 import native as nv

    precision = nv.HBG_MIXED if form == "mixed" else nv.HBG_FP64
    large = meshes.cylinder(1.0, 0.5, 64, 32, 32)  # 4096 panels
    small = meshes.cylinder(1.0, 0.5, 16, 8, 7)    # 240
    om = lambda n: np.sqrt(np.linspace(0.2, 1.2, n) * meshes.GRAVITY)  # noqa: E731
    few, many = om(8), om(2040)
    nv.lib().hbg_release_workspace()
    ref = nv.solve(small, many, [20.0], depth=5.0, precision=precision)
    nv.lib().hbg_release_workspace()
    nv.solve(large, om(12), (), depth=5.0, precision=nv.HBG_FP64)  # matrices of the other form held as well
    nv.solve(large, few, (), depth=5.0, precision=precision)
    fill = torch.empty(torch.cuda.mem_get_info()[0] - int(free_gb * 2 ** 30), dtype=torch.uint8, device="cuda")
    try:
        got = nv.solve(small, many, [20.0], depth=5.0, precision=precision)
        again = nv.solve(small, many, [20.0], depth=5.0, precision=precision)
    finally:
        del fill
        torch.cuda.empty_cache()
        nv.lib().hbg_release_workspace()
    for r in (got, again):
        for q in ("A", "B", "X"):  # the batches differ, and with them the number of corrections: the refinement's 1e-9 of
            a, b = np.asarray(r[q]), np.asarray(ref[q])  # the solution is 1e-7 of every entry's matrix and to spare
            assert np.abs(a - b).max() <= 1e-7 * np.abs(b).max(), q
