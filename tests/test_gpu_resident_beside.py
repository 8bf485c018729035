"""The one-kernel CG waits inside the kernel, so it has to get on beside other
work on the GPU: solves of several host threads at once, on streams of the
library's or the caller's, beside a stream kept busy with another library's
kernels.  Every result has the bits that the solve has alone."""
import threading

import numpy as np
import pytest

import fast_gb300 as ft
from fast_gb300 import _native, volumes

pytestmark = pytest.mark.gpu


def _solve(mask, prec, stream=None):
    import torch

    p = ft.TortuosityParams(tolerance=1e-9 if prec == ft.Precision.F64 else 1e-5, precision=prec)
    if stream is None:
        r = ft.solve_directions(mask, [ft.Dir.X_POS, ft.Dir.Z_NEG], p, ft.DSOLVER_CG)
    else:
        with torch.cuda.stream(stream):
            d = torch.from_numpy(mask).cuda()
        stream.synchronize()
        r = ft.solve_directions_device(d.data_ptr(), mask.shape, [ft.Dir.X_POS, ft.Dir.Z_NEG], p, ft.DSOLVER_CG,
                                       stream=stream.cuda_stream)
    assert _native.last_stats()["graph_replays"] == 0  # one kernel ran the iterations
    return [(x.tau, x.iterations, int(x.status)) for x in r]


def test_threads_and_a_busy_stream(gpu):
    import torch

    jobs = [(volumes.spheres(s, seed=k, r_min=2.0, solid_fraction=0.5), prec)
            for k, (s, prec) in enumerate([((20, 24, 28), ft.Precision.F64), ((48, 48, 48), ft.Precision.F64),
                                           ((40, 50, 64), ft.Precision.F32), ((64, 64, 64), ft.Precision.F32)])]
    alone = [_solve(m, p) for m, p in jobs]
    errors, done = [], threading.Event()

    def busy():
        st = torch.cuda.Stream()
        a = torch.rand(4 << 20, device="cuda")
        while not done.is_set():
            with torch.cuda.stream(st):
                for _ in range(20):
                    a = torch.sin(a) + 0.5
            st.synchronize()

    def solver(k):
        try:
            stream = torch.cuda.Stream() if k % 2 else None
            for _ in range(6):
                got = _solve(*jobs[k], stream=stream)
                if got != alone[k]:
                    errors.append((k, got, alone[k]))
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append((k, repr(e)))

    other = threading.Thread(target=busy)
    other.start()
    threads = [threading.Thread(target=solver, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    done.set()
    other.join()
    assert not errors
    assert np.all([a[2] == 0 for rows in alone for a in rows])
