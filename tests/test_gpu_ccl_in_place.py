"""Labels written over the mask they are made from (the mask in the first, the
last or a middle quarter of the labels' memory, or overlapping its end) equal
those of a mask of its own."""
import pytest

from fast_gb300 import ccl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(300, 90, 130), (9, 40, 65), (2, 3, 5)], ids=str)
@pytest.mark.parametrize("where", ["first", "middle", "last", "end"])
def test_mask_inside_the_labels(gpu, shape, where):
    import torch

    n = shape[0] * shape[1] * shape[2]
    gen = torch.Generator(device="cuda").manual_seed(n)
    mask = torch.where(torch.rand(shape, device="cuda", generator=gen) < 0.6, 255, 0).to(torch.uint8)
    want = torch.empty(shape, dtype=torch.int32, device="cuda")
    a = ccl.get_volume_ccl_device(mask.data_ptr(), shape, want.data_ptr())
    buf = torch.zeros(5 * n, dtype=torch.uint8, device="cuda")
    at = {"first": 0, "middle": n + 1, "last": 3 * n, "end": 4 * n - n // 2}[where]
    buf[at:at + n] = mask.flatten()
    torch.cuda.synchronize()
    b = ccl.get_volume_ccl_device(buf.data_ptr() + at, shape, buf.data_ptr())
    assert a.num_labels == b.num_labels and (a.boundary_label_mask == b.boundary_label_mask).all()
    assert torch.equal(buf[:4 * n].view(torch.int32), want.flatten())
