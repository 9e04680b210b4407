"""Bounded waits of the on-chip PCG kernels, each made to run out without a GPU
fault: with a short limit and an arrival that no block makes, every sum of a
team is waited for in vain, the kernels return, the solves report TIMEOUT and
leave the state, and the context goes on as before once the limit is back."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_team import _conf

pytestmark = pytest.mark.gpu

TINY = [(3 + k % 5, 4 + k % 3) for k in range(160)]  # more cloths than SMs


def _cloths(ctx, shapes, model):
    from acousticsim_gb300 import BaraffClothGpu
    out = []
    for k, (h, w) in enumerate(shapes):
        c = BaraffClothGpu(ctx, _conf(h, w, model))
        g = np.random.default_rng(30 + k)
        x = c.GetInitPos() + g.normal(0, 2e-4, c.nv * 3)
        out.append((c, x, x - 2e-3 * g.normal(0, 1e-2, c.nv * 3)))
    return out


def _step(ctx, cloths, p):
    for c, x, xp in cloths:
        c.Reset()
        c.SetPos(x)
        c.SetPrePos(xp)
    return ctx.batch_step([c for c, _, _ in cloths], 0.0, p)


# a cluster of one block, clusters of 16 (z rows between blocks, idle blocks), with
# skew parts; teams over the GPU with the stored blocks on chip, and with the matrix
# in memory, up to eight rows a thread and more; clusters of several sizes side by
# side, the largest with their stored blocks alone
@pytest.mark.parametrize("shapes,model", [([(16, 16)], "quadratic"), ([(64, 64)], "quadratic"),
                                          ([(21, 31)], "quadratic"), ([(64, 64)], "dihedral"),
                                          ([(300, 300)], "quadratic"), ([(300, 300)], "dihedral"),
                                          ([(560, 560)], "quadratic"), ([(700, 700)], "quadratic"),
                                          (TINY + [(62, 61), (100, 100)], "quadratic")])
def test_waits_run_out_and_context_recovers(built, shapes, model):
    from acousticsim_gb300 import ClothContext, params
    p = params(max_iters=40, rel_tol=1e-6)
    ctx = ClothContext(0)
    cloths = _cloths(ctx, shapes, model)
    ok = _step(ctx, cloths, p)
    assert all(s["status"] in ("OK", "MAXITER") and s["solver"] == "persistent" for s in ok), ok
    x_ok = [c.GetPos() for c, _, _ in cloths]

    ctx.set_spin_limit(1000, 1)
    st = _step(ctx, cloths, p)
    # (a cloth that is solved at its start waits for nothing)
    assert all(s["status"] == "TIMEOUT" and s["iters"] <= 1
               for s, o in zip(st, ok) if o["iters"] > 0), st
    pins = [c.GetConstraintStaticVertices() for c, _, _ in cloths]
    for (c, x, _), s, pin in zip(cloths, st, pins):
        if s["status"] == "TIMEOUT":
            free = np.ones(c.nv, bool)
            free[pin] = False
            assert np.array_equal(c.GetPos().reshape(-1, 3)[free], x.reshape(-1, 3)[free])

    ctx.set_spin_limit(0, 0)
    st = _step(ctx, cloths, p)
    assert [(s["status"], s["iters"]) for s in st] == [(s["status"], s["iters"]) for s in ok]
    for (c, _, _), x in zip(cloths, x_ok):
        assert np.array_equal(c.GetPos(), x)
        c.close()
    ctx.close()


def test_served_request_times_out_and_server_goes_on(built):
    from acousticsim_gb300 import ClothContext, ClothServer, params
    p = params(max_iters=4000, rel_tol=1e-6)
    ctx = ClothContext(0)
    shapes = [(16, 16), (64, 64)]
    ref = []
    for c, x, xp in _cloths(ctx, shapes, "quadratic"):
        c.SetPos(x)
        c.SetPrePos(xp)
        assert c.UpdatePos(0.0, p)["status"] == "OK"
        ref.append(c.GetPos())
        c.close()
    srv = ClothServer(ctx, 1 << 30, 0, 8)
    cloths = _cloths(ctx, shapes, "quadratic")
    for c, x, xp in cloths:
        c.SetPos(x)
        c.SetPrePos(xp)
        srv.add(c, 0.0, p)
    srv.start()
    for polls, extra, want in ((1000, 1, "TIMEOUT"), (0, 0, "OK")):
        ctx.set_spin_limit(polls, extra)
        for i in range(len(cloths)):
            srv.submit(i, i)
        srv.drain(60.0)
        res = srv.poll()
        assert len(res) == len(cloths) and all(r["status"] == want for r in res), res
    for (c, _, _), x in zip(cloths, ref):
        assert np.array_equal(c.GetPos(), x)
    srv.close()
    for c, _, _ in cloths:
        c.close()
    ctx.close()
