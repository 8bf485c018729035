"""The depth of a CG launch far larger than any GPU's memory, where counts of
its blocks leave the integers: the table's, as any launch that the model has
no better depth for."""
import pytest

import fast_gb300 as ft
from fast_gb300 import autotune as at

TABLE = (2, 4, 8, 16, 32, 64, 128, 256)


@pytest.mark.parametrize("prec", at.PRECISIONS)
@pytest.mark.parametrize("shape", [(2 ** 30, 2 ** 30, 2 ** 30), (2 ** 20, 2 ** 30, 2 ** 33), (2 ** 50, 3, 3),
                                   (5, 2 ** 30, 2 ** 38), (2 ** 31, 2 ** 31, 2 ** 31)], ids=str)
def test_table_depth_beyond_any_memory(native, monkeypatch, shape, prec):
    monkeypatch.delenv("FAST_TAU_ZC", raising=False)
    depth = at.slab_depth(shape, 6, prec, ft.DSOLVER_CG)[0]
    assert depth == shape[0] < 8 or depth in TABLE


@pytest.mark.parametrize("prec", at.PRECISIONS)
def test_model_depth_up_to_the_largest_volumes(native, monkeypatch, prec):
    monkeypatch.delenv("FAST_TAU_ZC", raising=False)
    for shape in ((2048, 2048, 2048), (2 ** 30, 8, 64), (3, 2 ** 27, 64)):
        assert 1 <= at.slab_depth(shape, 1, prec, ft.DSOLVER_CG)[0] <= min(shape[0], 1024)
