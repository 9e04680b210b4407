"""Parameters given while the kernels of an earlier call are still running: those
kernels keep the ones they were started with."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_team import _conf

pytestmark = pytest.mark.gpu


def test_solve_right_behind_an_assembly(ctx):
    """The assembly decides with its own tolerance (1e-6) that the solve begins; the
    solve's, which any residual meets, then ends it after one iteration."""
    from acousticsim_gb300 import BaraffClothGpu, params
    c = BaraffClothGpu(ctx, _conf(512, 512, "quadratic"))
    x = c.GetInitPos() + np.random.default_rng(3).normal(0, 1e-3, c.nv * 3)
    for _ in range(5):
        c.Reset()
        c.SetPos(x)
        c.SetPrePos(x)
        assert c.UpdatePos(0.0, params(max_iters=3, rel_tol=1e-6))["iters"] == 3
        c.SetPos(x)
        c.assemble()
        st = c.solve(params(max_iters=50, rel_tol=0.0, abs_tol=1e6))
        assert st["status"] == "OK" and st["iters"] == 1, st
    c.close()
