"""Domain faces in the FP64 and FP32 sweeps: the diagonal of a voxel on a face
comes from a table by its missing neighbours, so the shapes here have every
set of them (one- and two-voxel axes, volumes one voxel past a 64 x 8 tile).
Tolerances are those of the parity tests: F64 CG and the oracle at tol 1e-10
differ only in rounding (1e-9 in tau, iterations within 2), F32 at tol 1e-5
1e-4.  A served F64 request equals the same volume solved alone."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import fast_gb300 as ft
from fast_gb300.serve import TauServer

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
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


SCRIPT = r"""
import json, os, sys
sys.path.insert(0, %(root)r)
import numpy as np
import fast_gb300 as ft
from fast_gb300 import volumes
out = []
for shape in ((72, 70, 130), (33, 72, 200)):
    m = volumes.spheres(shape, seed=8, r_min=2.0, solid_fraction=0.5)
    nz, ny, nx = m.shape
    voxels = (nx + 15) // 16 * 16 * ny * nz
    for prec, size in ((ft.Precision.F64, 8), (ft.Precision.F32, 4)):
        row = []
        # room for everything, then for all but half of the stored product
        for free in (None, int(voxels * (4 * size + 1 + size / 2)) + 600000):
            os.environ.pop("FAST_TAU_TEST_FREE_BYTES", None)
            if free:
                os.environ["FAST_TAU_TEST_FREE_BYTES"] = str(free)
            it = []
            row.append([ft.get_tortuosity(m, ft.TortuosityParams(dir=ft.Dir.Y_POS, tolerance=1e-5, precision=prec),
                                          ft.DSOLVER_CG, iterations_out=it), it[0]])
        out.append(row)
print(json.dumps(out))
"""


def test_without_room_for_the_stored_product(gpu, tmp_path):
    """CG keeps q = A p where it fits; where it does not, step 2 evaluates
    the product again: the same bits."""
    code = ("import os, sys; sys.path.insert(0, %r)\n"
            "import fast_gb300.build as b\n"
            "b.OUT = %r; b.LIB = os.path.join(b.OUT, 'libfasttau.so'); b.CLI = os.path.join(b.OUT, 'fast')\n"
            "print(b.build(force=True))\n" % (ROOT, str(tmp_path)))
    env = dict(os.environ, FAST_TAU_NVCC_FLAGS="-DFAST_TAU_TEST_HOOKS=1")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, env=env, timeout=1800)
    assert r.returncode == 0, r.stderr[-2000:]
    env = dict(os.environ, FAST_TAU_LIB=r.stdout.strip().splitlines()[-1])
    r = subprocess.run([sys.executable, "-c", SCRIPT % {"root": ROOT}], capture_output=True, text=True, env=env,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    for stored, again in json.loads(r.stdout.strip().splitlines()[-1]):
        assert stored[0] > 0 and stored == again, (stored, again)
