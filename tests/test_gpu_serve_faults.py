"""A call that fails while a serving context starts its groups' chunks (a test
hook: after the first group's graph is launched, before the context's stream
waits for it).  The poll reports it; polled on, the context's requests end with
the results that each has alone; destroyed, it waits for what it launched."""
import json
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import json, os, sys
sys.path.insert(0, %(root)r)
import fast_gb300 as ft
from fast_gb300 import volumes
from fast_gb300.serve import TauServer

reqs = [(volumes.spheres(s, seed=k, r_min=3.0, solid_fraction=0.5), ft.Dir(k), solver)
        for k, (s, solver) in enumerate([((40, 64, 64), ft.DSOLVER_CG), ((64, 40, 64), ft.DSOLVER_BICGSTAB),
                                         ((50, 40, 95), ft.DSOLVER_CG)])]
alone = [ft.solve_directions(m, [d], ft.TortuosityParams(tolerance=1e-8), s)[0].tau for m, d, s in reqs]
out = {"alone": alone, "errors": []}

def failing_poll(srv):
    os.environ["FAST_TAU_TEST_FORK"] = "1"
    try:
        srv.poll()
    except RuntimeError as e:
        out["errors"].append(str(e))
    del os.environ["FAST_TAU_TEST_FORK"]

with TauServer(precision=ft.Precision.F64, tolerance=1e-8, chunk=2) as srv:
    for r in reqs:
        srv.submit(*r)
    failing_poll(srv)
    done = srv.poll()
    failing_poll(srv)
    done += srv.drain()
out["served"] = [c.result.tau for c in sorted(done, key=lambda c: c.ticket)]
with TauServer(precision=ft.Precision.F64, tolerance=1e-8, chunk=64) as srv:
    for r in reqs:
        srv.submit(*r)
    failing_poll(srv)
out["after"] = [ft.solve_directions(m, [d], ft.TortuosityParams(tolerance=1e-8), s)[0].tau for m, d, s in reqs]
print(json.dumps(out))
"""


def test_failing_fork(gpu, tmp_path):
    code = (
        "import os, sys; sys.path.insert(0, %r)\n"
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
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert len(out["errors"]) == 3 and all("FAST_TAU_TEST_FORK" in e for e in out["errors"])
    assert out["served"] == out["alone"] == out["after"]
