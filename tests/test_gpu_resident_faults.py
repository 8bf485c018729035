"""What goes wrong inside the one-kernel CG comes out of the call, in builds
with test hooks: a failed bounds check of its blocks (one checks an index of
an empty array, so nothing is accessed) fails the call as one in the sweeps
does; a block whose partial sum does not come (it publishes none in the third
iteration) makes the blocks that wait for it give up after the time limit, 50
ms here, and the call returns FAST_TIMEOUT.  Other right-hand sides of the
launch and the call after it are as before.  Where the cooperative launch is
refused, or the GPU has too few SMs for the blocks, the sweeps run instead:
the same bits, with the stored product that sweeps have."""
import json
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

pytestmark = pytest.mark.gpu

OK, CUDA_ERROR, TIMEOUT = 0, 6, 7

PRELUDE = r"""
import ctypes as C, json, os, sys
sys.path.insert(0, %(root)r)
import fast_gb300 as ft
from fast_gb300 import _native, volumes
L = _native.lib()
m = volumes.spheres((40, 36, 44), seed=8, r_min=3.0, solid_fraction=0.5)
nz, ny, nx = m.shape

def solve(dirs, prec, hook=None, arm=None, profile=False):
    for k in list(os.environ):
        if k.startswith("FAST_TAU_TEST_"):
            del os.environ[k]
    if hook:
        os.environ[hook] = str(arm)
    p = ft.TortuosityParams(tolerance=1e-8 if prec == ft.Precision.F64 else 1e-5, precision=prec,
                            profile=profile).to_c(ft.DSOLVER_CG)
    arr = (C.c_int32 * len(dirs))(*dirs)
    res = (_native.fast_tau_result * len(dirs))()
    st = L.fast_tau_solve_dirs(m.ctypes.data_as(C.c_void_p), nx, ny, nz, C.byref(p), len(dirs), arr, res)
    return [int(st), [[int(r.status), r.tau, int(r.iterations)] for r in res], _native.last_stats()["launches"],
            _native.last_error()]
"""


def _build(out, flags):
    code = (
        "import os, sys; sys.path.insert(0, %r)\n"
        "import fast_gb300.build as b\n"
        "b.OUT = %r; b.LIB = os.path.join(b.OUT, 'libfasttau.so'); b.CLI = os.path.join(b.OUT, 'fast')\n"
        "print(b.build(force=True))\n" % (ROOT, out))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True,
                       env=dict(os.environ, FAST_TAU_NVCC_FLAGS=flags), timeout=1800)
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout.strip().splitlines()[-1]


def _run(lib, body):
    r = subprocess.run([sys.executable, "-c", PRELUDE % {"root": ROOT} + body], capture_output=True, text=True,
                       env=dict(os.environ, FAST_TAU_LIB=lib), timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


BOUNDS = r"""
out = {}
for prec in (ft.Precision.F64, ft.Precision.F32):
    out[prec.name] = [solve([0, 2, 4], prec), solve([0, 2, 4], prec, "FAST_TAU_TEST_OOB", 3),
                      solve([0, 2, 4], prec), solve([0, 2, 4], prec, profile=True)]
print(json.dumps(out))
"""


def test_bounds_record_survives(gpu, tmp_path):
    lib = _build(str(tmp_path), "-DFAST_TAU_BOUNDS_CHECK=1 -DFAST_TAU_TEST_HOOKS=1")
    for before, armed, after, sweeps in _run(lib, BOUNDS).values():
        assert before[0] == after[0] == OK and before[1] == after[1]
        assert before[2] < sweeps[2]  # one kernel ran the iterations
        assert armed[0] == CUDA_ERROR and "bounds check" in armed[3]
        assert [r[0] for r in armed[1]] == [OK, CUDA_ERROR, OK] and armed[1][1][1] == 0.0
        assert armed[1][0] == before[1][0] and armed[1][2] == before[1][2]


SILENT = r"""
out = {}
for prec in (ft.Precision.F64, ft.Precision.F32):
    out[prec.name] = [solve([0, 2, 4], prec), solve([0, 2, 4], prec, "FAST_TAU_TEST_SILENT", 3),
                      solve([0, 2, 4], prec), solve([0, 2, 4], prec, profile=True)]
print(json.dumps(out))
"""


@pytest.fixture(scope="module")
def hooked_lib(tmp_path_factory):
    return _build(str(tmp_path_factory.mktemp("hooks")),
                  "-DFAST_TAU_TEST_HOOKS=1 -DFAST_TAU_WAIT_LIMIT_NS=50000000ull")


def test_missing_partial_sum_times_out(gpu, hooked_lib):
    for before, armed, after, sweeps in _run(hooked_lib, SILENT).values():
        assert before[0] == after[0] == OK and before[1] == after[1]
        assert before[2] < sweeps[2]  # one kernel ran the iterations
        assert armed[0] == TIMEOUT and "wait ran out" in armed[3] and "tile" not in armed[3]
        assert [r[0] for r in armed[1]] == [OK, TIMEOUT, OK] and armed[1][1][1] == 0.0
        assert armed[1][0] == before[1][0] and armed[1][2] == before[1][2]


REFUSED = r"""
def used_high(reset=False):  # bytes at most in use from the device's default memory pool
    cu, dev, pool, v = C.CDLL("libcuda.so.1"), C.c_int(), C.c_void_p(), C.c_uint64(0)
    assert cu.cuInit(0) == 0 and cu.cuDeviceGet(C.byref(dev), 0) == 0
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), dev) == 0
    if reset:
        assert cu.cuMemPoolSetAttribute(pool, 8, C.byref(v)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_HIGH
    assert cu.cuMemPoolGetAttribute(pool, 8, C.byref(v)) == 0
    return v.value

out = {}
for prec, n in ((ft.Precision.F64, 80), (ft.Precision.F32, 100)):
    m = volumes.spheres((n, n, n), seed=8, r_min=3.0, solid_fraction=0.5)
    nz, ny, nx = m.shape
    rows = []
    for kw in ({}, {"hook": "FAST_TAU_TEST_REFUSE", "arm": 1}, {"hook": "FAST_TAU_TEST_SMS", "arm": 8},
               {"profile": True}, {}):
        used_high(reset=True)
        rows.append(solve([2], prec, **kw) + [used_high()])
    out[prec.name] = rows
print(json.dumps(out))
"""


def test_refused_launch_runs_the_sweeps(gpu, hooked_lib):
    for kernel, refused, few_sms, sweeps, after in _run(hooked_lib, REFUSED).values():
        assert all(r[0] == OK for r in (kernel, refused, few_sms, sweeps, after))
        assert kernel[1] == refused[1] == after[1]
        assert refused[1] == sweeps[1]
        assert abs(few_sms[1][0][1] - kernel[1][0][1]) <= 1e-4 * kernel[1][0][1]  # another depth: other sums
        assert kernel[2] == after[2] < min(refused[2], few_sms[2], sweeps[2])
        assert refused[4] == sweeps[4] >= kernel[4] + (2 << 20)  # q: 4 MB
