"""CG of small FP64 and FP32 volumes in one kernel against the sweeps (which
profiles take): ragged tiles, slabs shorter than the others, one plane, one
row, many right-hand sides of which some end early, and sizes on both sides of
the rule.  The two do the same sums in the same order: FP64 tau within 1e-13
(rounding of fused and unfused products), FP32 within 1e-5, iterations within
2 (the bounds of the oracle's comparison)."""
import numpy as np
import pytest

import fast_gb300 as ft
from fast_gb300 import _native, volumes

pytestmark = pytest.mark.gpu


def _both(gpu, masks, dirs, prec, tol, max_iter=10000):
    out = []
    for profile in (False, True):
        p = ft.TortuosityParams(tolerance=tol, precision=prec, max_iter=max_iter, profile=profile)
        out.append(ft.solve_batch(list(zip(masks, dirs)), p, ft.DSOLVER_CG))
        out.append(_native.last_stats())
    return out


def _check(a, b, prec):
    for x, y in zip(a, b):
        assert x.status == y.status and abs(x.iterations - y.iterations) <= 2
        if x.status == 0:
            assert abs(x.tau - y.tau) <= (1e-13 if prec == ft.Precision.F64 else 1e-5) * y.tau


@pytest.mark.parametrize("prec", [ft.Precision.F64, ft.Precision.F32], ids=["f64", "f32"])
@pytest.mark.parametrize("shape", [(1, 9, 12), (12, 1, 9), (9, 12, 1), (7, 8, 64), (10, 9, 65), (61, 23, 66),
                                   (64, 64, 64)], ids=str)
def test_matches_the_sweeps(gpu, shape, prec):
    mask = volumes.spheres(shape, seed=8, r_min=2.0, solid_fraction=0.4) if min(shape) > 8 else np.where(
        np.random.default_rng(3).random(shape) < 0.4, 255, 0).astype(np.uint8)
    dirs = [ft.Dir(d) for d in (0, 2, 4)]
    tol = 1e-10 if prec == ft.Precision.F64 else 1e-5
    a, sa, b, sb = _both(gpu, [mask] * 3, dirs, prec, tol)
    assert sa["launches"] < sb["launches"]  # one kernel ran many iterations
    _check(a, b, prec)


def test_right_hand_sides_end_by_themselves(gpu):
    shapes = [(20, 24, 28), (5, 6, 7), (30, 17, 40), (1, 1, 3), (16, 16, 16)]
    masks = [np.where(np.random.default_rng(k).random(s) < 0.4, 255, 0).astype(np.uint8) for k, s in enumerate(shapes)]
    dirs = [ft.Dir(d) for d in (0, 3, 5, 1, 2)]
    a, sa, b, sb = _both(gpu, masks, dirs, ft.Precision.F64, 1e-10)
    assert sa["launches"] < sb["launches"]
    _check(a, b, ft.Precision.F64)
    a, _, b, _ = _both(gpu, masks, dirs, ft.Precision.F64, 1e-10, max_iter=3)  # and at the iteration limit
    _check(a, b, ft.Precision.F64)


def test_several_launches(gpu):
    mask = volumes.spheres((48, 48, 48), seed=8, r_min=2.0, solid_fraction=0.6)
    a, sa, b, _ = _both(gpu, [mask], [ft.Dir(0)], ft.Precision.F64, 1e-12)
    assert a[0].iterations > 128
    _check(a, b, ft.Precision.F64)
