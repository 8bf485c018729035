"""Labelling at the edges of its bricks (64 x 8 x 8 voxels, a row per 64-bit
word): sizes on both sides of a brick and of a word, dense and sparse noise,
a corridor that winds through every brick (the longest chains of joins) and
alternating voxels (as many runs as a word holds).  Bit-exact."""
import numpy as np
import pytest

from fast_gb300 import ccl

pytestmark = pytest.mark.gpu

SHAPES = [(8, 8, 64), (9, 9, 65), (7, 7, 63), (17, 16, 129), (1, 1, 200), (16, 1, 128), (1, 24, 1), (33, 40, 3)]


def _check(oracle, m, background=255):
    got = ccl.get_volume_ccl(m, background=background)
    labels, n = oracle.ccl_label(m, background=background)
    assert got.num_labels == n
    np.testing.assert_array_equal(got.labels, labels)
    np.testing.assert_array_equal(got.boundary_label_mask, oracle.ccl_boundary(labels, n))


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("pore", [0.1, 0.32, 0.5, 0.95])
def test_noise(gpu, oracle, shape, pore):
    m = np.where(np.random.default_rng(sum(shape)).random(shape) < pore, 0, 255).astype(np.uint8)
    _check(oracle, m)


def _corridor(nz, ny, nx):
    """One pore corridor along x in every other row, joined at alternating
    ends, the planes likewise."""
    m = np.full((nz, ny, nx), 255, np.uint8)
    rows = [(z, y) for k, z in enumerate(range(0, nz, 2)) for y in (range(0, ny, 2) if k % 2 == 0
                                                                    else range((ny - 1) // 2 * 2, -1, -2))]
    for k, (z, y) in enumerate(rows):
        m[z, y, :] = 0
        if k + 1 < len(rows):
            z2, y2 = rows[k + 1]
            m[(z + z2) // 2, (y + y2) // 2, nx - 1 if k % 2 == 0 else 0] = 0
    return m


@pytest.mark.parametrize("shape", [(17, 17, 130), (16, 24, 64)], ids=str)
def test_winding_corridor(gpu, oracle, shape):
    m = _corridor(*shape)
    assert oracle.ccl_label(m)[1] == 2  # one component
    for _ in range(3):
        _check(oracle, m)


def test_alternating_voxels(gpu, oracle):
    m = np.full((10, 11, 131), 255, np.uint8)
    m[:, :, ::2] = 0  # 32 runs a word, joined across y and z
    _check(oracle, m)
    m[::2] = 255
    _check(oracle, m, background=0)
