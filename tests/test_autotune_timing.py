"""What the autotuner times is what an installed table runs: launches at the
candidate depth by a table, not by the override that also fixes the tiles."""
import os

import fast_gb300 as ft
from fast_gb300 import autotune as at


def test_candidates_run_as_installed(native, monkeypatch):
    monkeypatch.setenv("FAST_TAU_ZC", "11")
    seen = []

    def timed(mask, dirs, prec, solver, iters):
        seen.append((os.environ.get("FAST_TAU_ZC"), at.slab_depth((66, 66, 66), 1, prec, solver)[0]))
        return 1.0, True

    monkeypatch.setattr(at, "_timed", timed)
    at._per_iteration(None, None, ft.Precision.F64, ft.DSOLVER_CG, 4, 8, 16, 1)
    assert seen == [(None, 4)] * 3
    assert os.environ["FAST_TAU_ZC"] == "11"
    monkeypatch.delenv("FAST_TAU_ZC")
    at.set_slab_table(ft.Precision.F64, ft.DSOLVER_CG, None)
    built_in = at.slab_depth((66, 66, 66), 1, ft.Precision.F64, ft.DSOLVER_CG)

    def failing(*args):
        raise RuntimeError("a solve that fails")

    monkeypatch.setattr(at, "_timed", failing)
    try:
        at._per_iteration(None, None, ft.Precision.F64, ft.DSOLVER_CG, 4, 8, 16, 1)
    except RuntimeError:
        pass
    assert at.slab_depth((66, 66, 66), 1, ft.Precision.F64, ft.DSOLVER_CG) == built_in
