"""Systems that FP32 does not resolve: p.q cancels until its chunks' rounding leaves
nothing of it and the solve stalls.  Every PCG driver ends such a solve as NaN in the
same iteration (a rule on exact sums), and a step escalates it to FP64."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_indefinite import _conf

pytestmark = pytest.mark.gpu


def _step(ctx, solver, conf, noise, p):
    from acousticsim_gb300 import BaraffClothGpu
    ctx.set_solver(solver)
    c = BaraffClothGpu(ctx, conf)
    g = np.random.default_rng(1234)
    x = c.GetInitPos().reshape(-1, 3) + g.normal(0.0, noise, (c.nv, 3))
    c.SetPos(x.reshape(-1))
    c.SetPrePos((x - 2e-3 * g.normal(0.0, 1e-2, x.shape)).reshape(-1))
    st, out = c.UpdatePos(0.0, p), c.GetPos()
    c.close()
    return st, out


def _dihedral(n, kb):
    return dict(_conf(n, 1e3), cloth_bending_model="dihedral", cloth_bending_stiffness=[kb, kb])


# negative stretch stiffness in one block and in clusters; dihedral bending with the
# whole matrix on chip, with the stored blocks, and (512) in the older kernel
@pytest.mark.parametrize("conf,noise", [(_conf(20, -1000.0), 1e-3), (_conf(40, -90.0), 1e-3),
                                        (_conf(40, -1000.0), 1e-3), (_dihedral(192, 0.1), 2e-3),
                                        (_dihedral(256, 0.1), 4e-3), (_dihedral(384, 1e-3), 2e-3),
                                        (_dihedral(512, 1e-3), 1e-3)])
def test_drivers_end_the_solve_in_the_same_iteration(built, conf, noise):
    from acousticsim_gb300 import ClothContext, params
    ctx = ClothContext(0)
    ctx.set_escalation(False)
    p = params(max_iters=20000, rel_tol=1e-6)
    a, b = (_step(ctx, s, conf, noise, p)[0] for s in ("persistent", "graph_loop"))
    ctx.close()
    assert a["solver"] == "persistent" and b["solver"] == "graph_loop"
    assert a["status"] == b["status"] == "NAN", (a, b)
    assert a["iters"] == b["iters"]


@pytest.mark.parametrize("n,kb,noise", [(256, 0.1, 4e-3), (300, 0.1, 8e-3), (384, 1e-3, 2e-3)])
def test_on_chip_solve_that_stalls_is_escalated(built, n, kb, noise):
    from acousticsim_gb300 import ClothContext, params
    ctx = ClothContext(0)
    st, x = _step(ctx, "persistent", _dihedral(n, kb), noise, params(max_iters=20000, rel_tol=1e-6))
    ctx.close()
    assert st["status"] == "OK" and st["solver"] == "escalated_fp64", st
    assert st["rel_residual"] <= 1e-6 and np.isfinite(x).all()


# without tolerances a solve goes on past its end: the residual leaves FP32's range, and
# noise comes back.  A strip and a square, the older kernels among the drivers
@pytest.mark.parametrize("h,w,density", [(5, 122, 0.0125), (24, 24, 0.1)])
def test_residual_that_comes_back_from_zero(built, h, w, density):
    from acousticsim_gb300 import ClothContext, params
    conf = dict(_conf(2, 350.0), subdivision=[h - 1, w - 1], cloth_density=density,
                cloth_bending_model="dihedral", cloth_bending_stiffness=[3e-4, 3e-4])
    p = params(max_iters=6000, rel_tol=0.0, abs_tol=0.0)
    ctx = ClothContext(0)
    ctx.set_escalation(False)
    st = [_step(ctx, s, conf, 1e-3, p)[0] for s in ("persistent", "graph_loop")]
    assert st[0]["status"] == st[1]["status"] == "NAN", st
    assert st[0]["iters"] == st[1]["iters"]
    ctx.set_escalation(True)
    for s in ("persistent", "graph_loop", "persistent_1b"):
        assert _step(ctx, s, conf, 1e-3, p)[0]["status"] == "OK"
    ctx.close()
