"""The F64 and F32 CG sweeps, which profiles take at every size: step 2 on the
stored product against step 2 that evaluates it again (the same bits; how much
device memory each run had shows which it was), and 32 x 16 tiles against 64 x
8 ones (a fixed depth keeps those).  Volumes of several slabs, on tiles of
either width, whose last tile is ragged.  A bounds-checked build runs the same
sweeps without an access out of range.  Tolerances are those of the oracle's
comparison: F64 1e-9 in tau and iterations within 2, F32 1e-4."""
import json
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

pytestmark = pytest.mark.gpu

PRELUDE = r"""
import ctypes as C, json, os, sys
sys.path.insert(0, %(root)r)
import numpy as np
import fast_gb300 as ft
from fast_gb300 import _native, autotune

NARROW = [(70, 50, 90), (45, 32, 150), (60, 64, 65)]  # (nz, ny, nx)
WIDE = [(72, 70, 130), (70, 41, 120), (45, 33, 161)]

def used_high(reset=False):  # bytes at most in use from the device's default memory pool
    cu, dev, pool, v = C.CDLL("libcuda.so.1"), C.c_int(), C.c_void_p(), C.c_uint64(0)
    assert cu.cuInit(0) == 0 and cu.cuDeviceGet(C.byref(dev), 0) == 0
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), dev) == 0
    if reset:
        assert cu.cuMemPoolSetAttribute(pool, 8, C.byref(v)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_HIGH
    assert cu.cuMemPoolGetAttribute(pool, 8, C.byref(v)) == 0
    return v.value

def mask(shape):
    return np.where(np.random.default_rng(shape[2]).random(shape) < 0.3, 255, 0).astype(np.uint8)

def solve(m, d, prec, env={}, solver=ft.DSOLVER_CG):
    for k in ("FAST_TAU_ZC", "FAST_TAU_TEST_FREE_BYTES"):
        os.environ.pop(k, None)
    os.environ.update(env)
    p = ft.TortuosityParams(tolerance=1e-10 if prec == ft.Precision.F64 else 1e-5, precision=prec, profile=True)
    used_high(reset=True)
    r = ft.solve_directions(m, [d], p, solver)[0]
    s = _native.last_stats()["kernels"]
    return {"tau": r.tau, "iters": r.iterations, "status": int(r.status), "memory": used_high(),
            "cg1": s.get("cg1", {}).get("launches", 0), "cg2": s.get("cg2", {}).get("launches", 0)}
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


def _run(body, lib=None):
    env = dict(os.environ, FAST_TAU_LIB=lib) if lib else dict(os.environ)
    r = subprocess.run([sys.executable, "-c", PRELUDE % {"root": ROOT} + body], capture_output=True, text=True, env=env,
                       timeout=900)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


@pytest.fixture(scope="module")
def hooked_lib(tmp_path_factory):
    return _build(str(tmp_path_factory.mktemp("hooks")), "-DFAST_TAU_TEST_HOOKS=1")


STORED = r"""
out = []
for shape in NARROW + WIDE:
    m = mask(shape)
    nz, ny, nx = shape
    voxels = (nx + 15) // 16 * 16 * ny * nz
    for prec, size in ((ft.Precision.F64, 8), (ft.Precision.F32, 4)):
        # room for everything, then for all but half of the stored product
        tight = {"FAST_TAU_TEST_FREE_BYTES": str(int(voxels * (4 * size + 1 + size / 2)) + 600000)}
        a, b = solve(m, ft.Dir.Y_POS, prec), solve(m, ft.Dir.Y_POS, prec, tight)
        out.append([shape, size * voxels, a, b])
print(json.dumps(out))
"""


def test_stored_product_against_evaluated_again(gpu, hooked_lib):
    for shape, q, stored, again in _run(STORED, hooked_lib):
        assert stored["status"] == again["status"] == 0
        assert stored["cg1"] >= stored["iters"] and stored["cg2"] >= stored["iters"]  # sweeps
        assert stored["memory"] - again["memory"] >= q  # q was there, and was not
        assert (stored["tau"], stored["iters"]) == (again["tau"], again["iters"]), shape


BESIDE = r"""
shape = (72, 70, 130)
m = mask(shape)
nz, ny, nx = shape
voxels = (nx + 15) // 16 * 16 * ny * nz
need = voxels * 33  # four vectors and the codes, and 4 % for all else
q = voxels * 8
out = [q]
for free in (1.04 * need + q, 2.08 * need + q / 2, 2.08 * need + 1.1 * q):
    out.append(solve(m, ft.Dir.Y_POS, ft.Precision.F64, {"FAST_TAU_TEST_FREE_BYTES": str(int(free))}))
print(json.dumps(out))
"""


def test_stored_product_leaves_room_for_a_second_solve(gpu, hooked_lib):
    """No second solve of the size fits; one fits beside the plain plan alone;
    one fits beside q too."""
    q, filled, beside, roomy = _run(BESIDE, hooked_lib)
    assert filled["memory"] == roomy["memory"] >= beside["memory"] + q
    assert filled["tau"] == beside["tau"] == roomy["tau"]


TILES = r"""
out = []
for shape in NARROW:
    m = mask(shape)
    for prec in (ft.Precision.F64, ft.Precision.F32):
        for d in (ft.Dir(0), ft.Dir(3), ft.Dir(4)):
            for zc in (str(autotune.slab_depth(shape, 1, prec, ft.DSOLVER_CG)[0]), "16"):
                out.append([list(shape), int(prec), int(zc), solve(m, d, prec), solve(m, d, prec, {"FAST_TAU_ZC": zc})])
print(json.dumps(out))
"""


def test_narrow_sweeps_match_the_wide_ones(gpu):
    for (nz, ny, nx), prec, zc, narrow, wide in _run(TILES):
        tiles = [-(-nx // w) * -(-ny // (512 // w)) for w in (32, 64)]
        assert 100 * tiles[0] <= 97 * tiles[1] and zc < nz  # the rule's width; several slabs
        for r in (narrow, wide):
            assert r["status"] == 0 and r["cg1"] >= r["iters"] and r["cg2"] >= r["iters"]
        assert abs(narrow["tau"] - wide["tau"]) <= (1e-9 if prec == 0 else 1e-4) * wide["tau"]
        assert prec != 0 or abs(narrow["iters"] - wide["iters"]) <= 2


BOUNDS = r"""
out = []
for shape in NARROW + WIDE:
    m = mask(shape)
    for prec in (ft.Precision.F64, ft.Precision.F32):
        for env in ({}, {"FAST_TAU_ZC": "7"}):
            for solver in (ft.DSOLVER_CG, ft.DSOLVER_BICGSTAB):
                r = solve(m, ft.Dir.Z_NEG, prec, env, solver)
                out.append([r["tau"], r["iters"], r["status"]])
print(json.dumps(out))
"""


def test_no_access_out_of_range(gpu, tmp_path):
    checked = _run(BOUNDS, _build(str(tmp_path), "-DFAST_TAU_BOUNDS_CHECK=1"))
    assert checked == _run(BOUNDS)
    assert all(r[2] == 0 for r in checked[::2])  # CG
