"""Labelling of the longest rows the entry point takes (2^31 - 1 voxels on an
axis, where one brick more would leave 32-bit coordinates): a few components,
the last at the very end, as a row and as a column."""
import numpy as np
import pytest

from fast_gb300 import ccl

pytestmark = pytest.mark.gpu

N = 2 ** 31 - 1


@pytest.mark.parametrize("shape", [(1, 1, N), (1, N, 1), (N, 1, 1)], ids=["x", "y", "z"])
def test_longest_axis(gpu, shape):
    import torch

    mask = torch.full((N,), 255, dtype=torch.uint8, device="cuda")
    spans = [(0, 1), (5, 70), (N // 2, N // 2 + 1000), (N - 65, N - 64), (N - 3, N)]
    for a, b in spans:
        mask[a:b] = 0
    labels = torch.empty(N, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    got = ccl.get_volume_ccl_device(mask.data_ptr(), shape, labels.data_ptr())
    assert got.num_labels == len(spans) + 1
    for k, (a, b) in enumerate(spans):
        assert bool((labels[a:b] == k + 1).all())
    assert int((labels != 0).sum(dtype=torch.int64)) == sum(b - a for a, b in spans)
    axis = [2, 1, 0][[i for i in range(3) if shape[i] == N][0]]
    rows = np.ones((6, got.num_labels), np.uint8)
    rows[:, 0] = 0
    rows[2 * axis] = [0, 0, 0, 0, 0, 1]
    rows[2 * axis + 1] = [0, 1, 0, 0, 0, 0]
    assert (got.boundary_label_mask[:6] == rows).all()
    del mask, labels
    torch.cuda.empty_cache()
