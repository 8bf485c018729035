"""The area pass adds in double: where the triangles' areas are such that every
partial sum fits a double (all are multiples of the last bit of the smallest
one, and their sum is below 2^53 of those), the area is their exact sum,
whatever the order.  An isovalue just below 1/8 puts vertices next to the grid
points, so that the areas of a few cells span more than 2^20 and a sum in
fewer bits has to round."""
import ctypes as C
import math

import numpy as np
import pytest

from fast_gb300 import Status

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [8, 64, 1024, 4096])
def test_exact_where_a_double_is(gpu, oracle, nz):
    rng = np.random.default_rng(nz)
    iso, held = 0.1249, 0
    for _ in range(60):
        ny, nx = int(rng.integers(1, 4)), int(rng.integers(2, 5))
        m = np.zeros((nz, ny, nx), np.uint8)
        m[:12] = np.where(rng.random(m[:12].shape) < 0.3, 255, 0)
        area, low, smallest = oracle.area_sum(m, iso)
        last_bit = math.ldexp(1.0, math.frexp(smallest)[1] - 24) if math.isfinite(smallest) else 1.0
        if low != 0.0 or area >= 2.0 ** 53 * last_bit:
            continue
        held += 1
        out = C.c_double()
        st = gpu.fast_reactive_area(m.ctypes.data_as(C.c_void_p), nx, ny, nz, iso, C.byref(out))
        assert st == Status.OK, gpu.fast_last_error()
        assert out.value == area
    assert held >= 30
