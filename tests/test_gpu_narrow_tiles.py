"""CG on 32 x 16 tiles (taken where they cover a volume with fewer tiles)
against 64 x 8 ones (a fixed depth keeps them): widths and heights at the edges
of both tiles, every precision, batches that mix them, and served requests of
both kinds.  Tolerances are those of the oracle's comparison: the two sum in
another order (F64 1e-9 in tau and iterations within 2, F32 1e-4, MIXED 1e-5)."""
import numpy as np
import pytest

import fast_gb300 as ft
from fast_gb300 import autotune, volumes
from fast_gb300.serve import TauServer

pytestmark = pytest.mark.gpu

SHAPES = [(3, 16, 1), (20, 24, 28), (9, 33, 31), (12, 32, 32), (17, 9, 65), (30, 16, 70), (40, 50, 95), (33, 15, 96),
          (21, 49, 97), (70, 80, 150)]
TOL = {ft.Precision.F64: (1e-10, 1e-9), ft.Precision.F32: (1e-5, 1e-4), ft.Precision.MIXED: (1e-7, 1e-5)}


def _mask(shape):
    return np.where(np.random.default_rng(shape[2]).random(shape) < 0.3, 255, 0).astype(np.uint8)


@pytest.mark.parametrize("prec", list(TOL), ids=str)
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_matches_the_wide_tiles(gpu, monkeypatch, shape, prec):
    tol, bound = TOL[prec]
    mask = _mask(shape)
    for d in (0, 3, 4):
        p = ft.TortuosityParams(dir=ft.Dir(d), tolerance=tol, precision=prec)
        got = {}
        for zc in ("", str(autotune.slab_depth(shape, 1, prec, ft.DSOLVER_CG)[0])):
            it = []
            monkeypatch.setenv("FAST_TAU_ZC", zc) if zc else monkeypatch.delenv("FAST_TAU_ZC", raising=False)
            got[bool(zc)] = ft.get_tortuosity(mask, p, ft.DSOLVER_CG, iterations_out=it), it[0]
        monkeypatch.delenv("FAST_TAU_ZC", raising=False)
        (a, ia), (b, ib) = got[False], got[True]
        assert abs(a - b) <= bound * abs(b)
        if prec == ft.Precision.F64:
            assert abs(ia - ib) <= 2


@pytest.mark.parametrize("prec", [ft.Precision.F64, ft.Precision.MIXED], ids=str)
def test_batch_and_serving(gpu, prec):
    tol, bound = TOL[prec]
    masks = [_mask(s) for s in ((20, 24, 28), (30, 16, 64), (40, 50, 95), (25, 40, 128))]
    p = ft.TortuosityParams(dir=ft.Dir(0), tolerance=tol, precision=prec)
    alone = [ft.get_tortuosity(m, p, ft.DSOLVER_CG) for m in masks]
    batch = ft.solve_batch([(m, ft.Dir(0)) for m in masks], p, ft.DSOLVER_CG)
    for r, t in zip(batch, alone):
        assert r.status == 0 and abs(r.tau - t) <= bound * t
    with TauServer(precision=prec, tolerance=tol, chunk=8) as srv:
        for m in masks:
            srv.submit(m, ft.Dir(0), ft.DSOLVER_CG)
        srv.submit(masks[0], ft.Dir(0), ft.DSOLVER_BICGSTAB)
        done = sorted(srv.drain(), key=lambda c: c.ticket)
    assert [c.result.tau for c in done[:4]] == alone
    assert done[4].result.status == 0
