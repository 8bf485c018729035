"""The area pass at the edges of its bricks (62 x 16 x up to 16 cells, 64
voxels in a word): sizes on both sides of a brick, a volume large enough for
the deepest bricks with nearly every cell cut (more cells than the queue
holds at once), and noise whose components touch every mixture of faces.
The oracle evaluates each triangle in the same float sequence; the sums differ
in order and in the last bits of a pair sum (2^-47) or a double, so 1e-11."""
import ctypes as C

import numpy as np
import pytest

from fast_gb300 import Status

pytestmark = pytest.mark.gpu


def _noise(shape, solid, seed):
    return np.where(np.random.default_rng(seed).random(shape) < solid, 255, 0).astype(np.uint8)


def _tensor(gpu, m, iso):
    nz, ny, nx = m.shape
    t, solid = (C.c_double * 6)(), C.c_double()
    st = gpu.fast_reactive_area_tensor(m.ctypes.data_as(C.c_void_p), nx, ny, nz, iso, t, C.byref(solid))
    assert st == Status.OK, gpu.fast_last_error()
    return list(t), solid.value


def _close(a, b):
    return abs(a - b) <= 1e-11 * abs(b) or abs(a - b) < 1e-14


@pytest.mark.parametrize("shape", [(16, 16, 62), (17, 17, 63), (15, 33, 61), (2, 1, 125), (33, 2, 64)], ids=str)
@pytest.mark.parametrize("iso", [0.0, 0.125, 0.5, 1.0, 1.5])
def test_brick_edges(gpu, oracle, shape, iso):
    m = _noise(shape, 0.62, 3)
    t, area = _tensor(gpu, m, iso)
    want = oracle.reactive_area_tensor(m, iso)
    assert _close(area, oracle.reactive_area(m, iso))
    for d in range(6):
        assert _close(t[d], want[d]), d


def test_deep_bricks_with_nearly_every_cell_cut(gpu, oracle):
    m = _noise((258, 250, 249), 0.5, 4)
    nz, ny, nx = m.shape
    out = C.c_double()
    st = gpu.fast_reactive_area(m.ctypes.data_as(C.c_void_p), nx, ny, nz, 0.5, C.byref(out))
    assert st == Status.OK, gpu.fast_last_error()
    assert _close(out.value, oracle.reactive_area(m, 0.5))
