"""The area pass on the longest axes the entry point takes (2^31 - 1 voxels,
where coordinates beside a brick leave 32 bits).  A row of voxels across an
axis has one face of area 1 wherever solid and pore meet, so the areas are
counts of those; the labels of the pores name the faces they touch."""
import ctypes as C

import pytest

from fast_gb300 import Status

pytestmark = pytest.mark.gpu

N = 2 ** 31 - 1


@pytest.mark.parametrize("axis", [0, 1, 2], ids=["x", "y", "z"])
def test_longest_axis(gpu, axis):
    import torch

    dims = [1, 1, 1]
    dims[axis] = N
    mask = torch.zeros(N, dtype=torch.uint8, device="cuda")
    mask[10:200] = 255
    mask[N // 2:N // 2 + 7] = 255
    mask[N - 60:] = 255
    torch.cuda.synchronize()
    area, tensor = C.c_double(), (C.c_double * 6)()
    st = gpu.fast_reactive_area_device(C.c_void_p(mask.data_ptr()), *dims, 0.5, C.byref(area), None)
    assert st == Status.OK, gpu.fast_last_error()
    assert area.value == 5.0
    st = gpu.fast_reactive_area_tensor_device(C.c_void_p(mask.data_ptr()), *dims, 0.5, tensor, C.byref(area), None)
    assert st == Status.OK, gpu.fast_last_error()
    want = [5.0] * 6  # every pore touches the four long faces
    want[2 * axis], want[2 * axis + 1] = 0.0, 1.0  # none the far end, the first the near one
    assert list(tensor) == want and area.value == 5.0
    del mask
    torch.cuda.empty_cache()
