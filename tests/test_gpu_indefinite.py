"""Solves whose sums cancel: cloths of negative stretch stiffness, whose system is
indefinite.  Chunks of p.q are then up to hundreds of times p.q, which may grow
2^20-fold from one iteration to the next.  A sum is exact as long as it and its
chunks are in range, so each PCG driver takes the same iterations to the same
bits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _conf(n, k):
    return {"geometry_type": "regular_triangle", "cloth_size": [1.0, 1.0],
            "subdivision": [n - 1, n - 1], "cloth_init_pos": [0.0, 0.0, 0.0],
            "cloth_uv_rotation": 0, "cloth_stretch_stiffness": [k, k, k / 10],
            "cloth_bending_stiffness": [1e-3, 1e-3], "cloth_density": 0.1,
            "rayleigh_damping_a": 0.01, "rayleigh_damping_b": 0.0, "default_timestep": 2e-3,
            "constraints": {"static_point": [[-0.5, 0.5], [0.5, 0.5]]}}


def _step(ctx, solver, n, k, p):
    """One FP32 step of a seeded state by a driver: stats and positions."""
    from acousticsim_gb300 import BaraffClothGpu
    ctx.set_solver(solver)
    c = BaraffClothGpu(ctx, _conf(n, k))
    g = np.random.default_rng(1234)
    x = c.GetInitPos().reshape(-1, 3) + g.normal(0.0, 1e-3, (c.nv, 3))
    xp = x - 2e-3 * g.normal(0.0, 1e-2, x.shape)
    c.SetPos(x.reshape(-1))
    c.SetPrePos(xp.reshape(-1))
    st, out = c.UpdatePos(0.0, p), c.GetPos()
    c.close()
    return st, out


# one block, and clusters: chunks past the range that a sum itself may have
@pytest.mark.parametrize("n,k", [(16, -60.0), (20, -40.0), (24, -15.0)])
def test_indefinite_solve_converges_in_every_driver(built, n, k):
    from acousticsim_gb300 import ClothContext, params
    p = params(max_iters=2000, rel_tol=1e-5)
    ctx = ClothContext(0)
    ctx.set_escalation(False)
    out = {s: _step(ctx, s, n, k, p) for s in ("persistent", "graph_loop")}
    ctx.close()
    a, b = out["persistent"], out["graph_loop"]
    assert a[0]["solver"] == "persistent" and b[0]["solver"] == "graph_loop"
    assert a[0]["status"] == b[0]["status"] == "OK", (a[0], b[0])
    assert a[0]["iters"] == b[0]["iters"]
    assert np.array_equal(a[1], b[1])
