"""The depth a CG launch takes: the built-in table's, or an even split of the
tallest volume that a model of the GPU's waves of blocks puts well below it.
Launches whose blocks exceed one wave by little get the depth that fits; an
installed table and the override are followed; BiCGSTAB keeps the table."""
import pytest

import fast_gb300 as ft
from fast_gb300 import autotune as at

F64, F32, MIXED = ft.Precision.F64, ft.Precision.F32, ft.Precision.MIXED


@pytest.fixture
def clean(monkeypatch, native):
    monkeypatch.delenv("FAST_TAU_ZC", raising=False)
    for p in at.PRECISIONS:
        for s in at.SOLVERS:
            at.set_slab_table(p, s, None)
    yield
    for p in at.PRECISIONS:
        for s in at.SOLVERS:
            at.set_slab_table(p, s, None)


def _depth(shape, n, prec, solver=ft.DSOLVER_CG):
    return at.slab_depth(shape, n, prec, solver)[0]


@pytest.mark.parametrize("prec", [F64, F32, MIXED])
@pytest.mark.parametrize("shape,n", [((1, 1, 1), 1), ((2 ** 20, 3, 3), 1), ((97, 83, 110), 1), ((256, 256, 256), 3),
                                     ((1024, 1024, 1024), 1), ((5, 700, 900), 6)])
def test_depth_is_an_even_split_or_the_tables(clean, prec, shape, n):
    nz = shape[0]
    d = _depth(shape, n, prec)
    assert 1 <= d <= min(nz, 1024)
    at.set_slab_table(prec, ft.DSOLVER_CG, [7] * 32)  # an installed table is followed
    assert _depth(shape, n, prec) == min(7, nz)
    at.set_slab_table(prec, ft.DSOLVER_CG, None)
    if d not in (2, 4, 8, 16, 32, 64, 128, 256):
        assert -(-nz // -(-nz // d)) == d  # even slabs


def test_one_wave_where_the_table_needs_two(clean):
    # 256^3 in one direction: 128 columns of tiles; 8 slabs of 32 planes are
    # 1024 blocks where 912 are resident, 7 of 37 are 896
    assert _depth((256, 256, 256), 1, MIXED) == 37
    # F64, 304 resident: 96 columns of tiles in three directions
    assert _depth((128, 128, 128), 3, F64) == 43  # 3 slabs x 96 columns = 288


def test_bicgstab_keeps_the_table(clean):
    for prec in (F64, F32, MIXED):
        d = _depth((256, 256, 256), 1, prec, ft.DSOLVER_BICGSTAB)
        assert d in (2, 4, 8, 16, 32, 64, 128, 256)


def test_override(clean, monkeypatch):
    monkeypatch.setenv("FAST_TAU_ZC", "9")
    assert _depth((256, 256, 256), 1, MIXED) == 9
