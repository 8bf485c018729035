"""Domain faces in the FP64 and FP32 sweeps: the diagonal of a voxel on a face
comes from a table by its missing neighbours, so the shapes here have every
set of them (one- and two-voxel axes, volumes one voxel past a 64 x 8 tile).
Tolerances are those of the parity tests: F64 CG and the oracle at tol 1e-10
differ only in rounding (1e-9 in tau, iterations within 2), F32 at tol 1e-5
1e-4.  A served F64 request equals the same volume solved alone."""
import numpy as np
import pytest

import fast_gb300 as ft
from fast_gb300.serve import TauServer

pytestmark = pytest.mark.gpu

SHAPES = [(1, 9, 12), (12, 1, 9), (9, 12, 1), (2, 2, 2), (3, 2, 65), (10, 9, 66)]


def _mask(shape, seed):
    return np.where(np.random.default_rng(seed).random(shape) < 0.4, 255, 0).astype(np.uint8)


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_f64_and_f32_match_the_oracle(gpu, oracle, shape):
    mask = _mask(shape, 31)
    for d in range(6):
        it = []
        tau = ft.get_tortuosity(mask, ft.TortuosityParams(dir=ft.Dir(d), tolerance=1e-10), ft.DSOLVER_CG,
                                iterations_out=it)
        ref = oracle.get_tortuosity(mask, dir=d, solver=1, tol=1e-10)
        if ref["status"] != 0:  # a one-plane axis has no right-hand side in the negative direction
            assert tau == 0.0
            continue
        assert abs(tau - ref["tau"]) <= 1e-9 * ref["tau"] and abs(it[0] - ref["iters"]) <= 2
        tau = ft.get_tortuosity(mask, ft.TortuosityParams(dir=ft.Dir(d), tolerance=1e-10), ft.DSOLVER_BICGSTAB)
        assert abs(tau - ref["tau"]) <= 1e-8 * ref["tau"]
        tau = ft.get_tortuosity(mask, ft.TortuosityParams(dir=ft.Dir(d), tolerance=1e-5, precision=ft.Precision.F32),
                                ft.DSOLVER_CG)
        ref = oracle.get_tortuosity(mask, dir=d, solver=1, tol=1e-5, dtype=np.float32)
        assert abs(tau - ref["tau"]) <= 1e-4 * ref["tau"]


@pytest.mark.parametrize("precision", [ft.Precision.F64, ft.Precision.F32])
def test_served_alone(gpu, precision):
    mask = _mask((9, 10, 11), 5)
    with TauServer(precision=precision, tolerance=1e-5, max_inflight=1) as srv:
        for d in (0, 3, 5):
            srv.submit(mask, ft.Dir(d), ft.DSOLVER_CG)
        served = [c.result.tau for c in sorted(srv.drain(), key=lambda c: c.ticket)]
    alone = [ft.get_tortuosity(mask, ft.TortuosityParams(dir=ft.Dir(d), tolerance=1e-5, precision=precision),
                               ft.DSOLVER_CG) for d in (0, 3, 5)]
    assert served == alone
