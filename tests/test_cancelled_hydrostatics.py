"""A solve of the FP64 form that is cancelled before its first batch has still written the hydrostatics."""
from __future__ import annotations

import ctypes
import math

import numpy as np
import pytest

from hydrobem_b200 import meshes


@pytest.mark.gpu
def test_hydrostatics_of_a_cancelled_solve():
    from hydrobem_b200 import native as nv

    v = meshes.cylinder(1.0, 0.5, 16, 4, 4)
    body = nv.Body(v, [1.0, 2.0], [20.0])
    flag = ctypes.c_int32(1)
    field = dict(nv.HbgOptions._fields_)["cancel"]
    with pytest.raises(nv.HydroBEMError, match="cancelled"):
        nv.solve_batch([body], depth=math.inf, precision=nv.HBG_FP64, cancel=ctypes.cast(ctypes.pointer(flag), field))
    ref = nv.Body(v, [])
    nv.solve_batch([ref], depth=math.inf, precision=nv.HBG_FP64)
    assert ref.HS[0, 0] > 1.0 and np.array_equal(body.HS, ref.HS, equal_nan=True)  # (no mass given: NaN)
