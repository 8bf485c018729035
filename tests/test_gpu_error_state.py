"""A call that fails because the GPU's memory does not hold what it asks for
leaves nothing behind: the calls after it succeed.  (The volume of the failing
call is described, not there: the call ends at its allocation.)"""
import ctypes as C

import numpy as np
import pytest

import fast_gb300 as ft
from fast_gb300 import Status, _native, alpha, ccl, volumes
from fast_gb300.serve import TauServer

pytestmark = pytest.mark.gpu


def _fails(gpu, mask):
    v = (_native.fast_tau_volume * 1)()
    v[0].mask = mask.ctypes.data_as(C.c_void_p)
    v[0].nx = v[0].ny = v[0].nz = 1 << 20  # 2^60 bytes
    p = ft.TortuosityParams().to_c(ft.DSOLVER_CG)
    res = (_native.fast_tau_result * 1)()
    assert gpu.fast_tau_solve_batch(v, 1, C.byref(p), res) == Status.NOMEM


def test_next_call_succeeds(gpu):
    m = volumes.spheres((12, 14, 16), seed=3, r_min=2.0, solid_fraction=0.4)
    _fails(gpu, m)
    assert ft.get_porosity(m) == np.count_nonzero(m == 0) / m.size
    _fails(gpu, m)
    with TauServer(max_inflight=1) as srv:
        srv.submit(m, ft.Dir.X_POS, ft.DSOLVER_CG)
        assert srv.drain()[0].result.status == ft.Status.OK
    _fails(gpu, m)
    assert ccl.get_volume_ccl(m).num_labels > 1
    _fails(gpu, m)
    assert alpha.get_reactive_area_density(m) > 0.0
    _fails(gpu, m)
    assert ft.get_tortuosity(m, ft.TortuosityParams(dir=ft.Dir.X_POS), ft.DSOLVER_CG) > 1.0
