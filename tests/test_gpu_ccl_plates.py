"""Rows that all look alike: plates and columns across x, whose runs start at
the same places in every row of a brick (up to the 32 of a word), with the
plates joined at one corner, one edge, or not at all."""
import numpy as np
import pytest

from fast_gb300 import ccl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("period", [2, 3, 4, 64])
@pytest.mark.parametrize("join", ["none", "corner", "edge"])
def test_plates(gpu, oracle, period, join):
    m = np.full((19, 21, 150), 255, np.uint8)
    m[:, :, ::period] = 0
    if join == "corner":
        m[18, 20, :] = 0
    elif join == "edge":
        m[9, :, :] = 0
    got = ccl.get_volume_ccl(m)
    want, n = oracle.ccl_label(m, 255)
    assert got.num_labels == n and np.array_equal(got.labels, want)
    columns = m.copy()
    columns[:, ::2, :] = 255
    got = ccl.get_volume_ccl(columns)
    want, n = oracle.ccl_label(columns, 255)
    assert got.num_labels == n and np.array_equal(got.labels, want)
