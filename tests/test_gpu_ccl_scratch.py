"""Scratch memory of a labelling, as the device's memory pool counts it: no
width from 4 voxels on takes more than the 4.125 bytes per voxel (and 2 MB of
rounding) that a parent per voxel took, nor does one voxel, whose labels and
faces equal the oracle's."""
import ctypes as C

import numpy as np
import pytest

from fast_gb300 import ccl

pytestmark = pytest.mark.gpu


def _used_high(reset=False):
    cu, dev, pool, v = C.CDLL("libcuda.so.1"), C.c_int(), C.c_void_p(), C.c_uint64(0)
    assert cu.cuInit(0) == 0 and cu.cuDeviceGet(C.byref(dev), 0) == 0
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), dev) == 0
    if reset:
        assert cu.cuMemPoolSetAttribute(pool, 8, C.byref(v)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_HIGH
    assert cu.cuMemPoolGetAttribute(pool, 8, C.byref(v)) == 0
    return v.value


@pytest.mark.parametrize("nx", [1, 4, 7, 33, 64, 65, 129])
def test_scratch_per_voxel(gpu, nx):
    import torch

    shape = (8000000 // (800 * nx), 800, nx)
    n = shape[0] * shape[1] * shape[2]
    gen = torch.Generator(device="cuda").manual_seed(nx)
    mask = torch.where(torch.rand(shape, device="cuda", generator=gen) < 0.5, 255, 0).to(torch.uint8)
    labels = torch.empty(shape, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    base = _used_high(reset=True)
    ccl.get_volume_ccl_device(mask.data_ptr(), shape, labels.data_ptr(), boundary=False)
    assert _used_high() - base <= 4.125 * n + (2 << 20)


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 70, 1), (130, 1, 1), (67, 129, 1), (9, 65, 1)], ids=str)
def test_one_voxel_wide(gpu, oracle, shape):
    m = np.where(np.random.default_rng(sum(shape)).random(shape) < 0.4, 255, 0).astype(np.uint8)
    got = ccl.get_volume_ccl(m)
    want, n = oracle.ccl_label(m, 255)
    assert got.num_labels == n and np.array_equal(got.labels, want)
    assert np.array_equal(got.boundary_label_mask, oracle.ccl_boundary(want, n))
