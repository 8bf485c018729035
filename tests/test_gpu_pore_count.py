"""fast_porosity counts a volume's zero bytes sixteen at a time: sizes on both
sides of a vector, of a block and of the resident grid, and bytes of every
value.  Counts are integers: equal."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 1, 15), (1, 1, 16), (1, 1, 17), (3, 37, 37), (1, 64, 64), (5, 1000, 1001),
                                   (1, 1216, 4099)], ids=str)
def test_counts(gpu, shape):
    rng = np.random.default_rng(sum(shape))
    for m in (rng.integers(0, 3, shape, dtype=np.uint8) * rng.integers(0, 256, shape, dtype=np.uint8),
              np.zeros(shape, np.uint8), np.full(shape, 128, np.uint8)):
        nz, ny, nx = shape
        phi, n = C.c_double(0), C.c_uint64(1)
        assert gpu.fast_porosity(m.ctypes.data_as(C.c_void_p), nx, ny, nz, C.byref(phi), C.byref(n)) == 0
        assert n.value == int((m == 0).sum()) and phi.value == n.value / m.size
