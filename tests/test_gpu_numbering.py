"""Meshes whose vertices are numbered in any order (an OBJ file's): a block's rows then
touch columns all over its cloth, and the solver plans differ.  Whatever kernel a plan
takes, its iterations and positions are the graph loop's bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_team import _conf

pytestmark = pytest.mark.gpu


def _mesh(h, w, within):
    """A grid whose vertices are moved up to `within` places in their order (0: not)."""
    from acousticsim_gb300.cloth import build_grid
    m = build_grid((1.0, 1.0), (h - 1, w - 1))
    if within == 0:
        return m
    pos = m["pos"].reshape(-1, 3)
    order = np.argsort(np.arange(len(pos)) + np.random.default_rng(5).uniform(0, within, len(pos)))
    place = np.argsort(order)
    return {"pos": pos[order], "uv": m["uv"].reshape(-1, 2)[order],
            "tris": place[m["tris"].reshape(-1, 3)].astype(np.int32)}


ANY = 10 ** 9


# a cluster of one block, of 16 (every block sends its rows to every other), the whole
# GPU with the whole matrix on chip; cloths of which a block touches most, and a third,
# with the matrix in memory; sets: clusters in one wave, one more cloth than run at once,
# many; in grid order, more cloths with stored blocks than run at once, with an idle last
# wave and with a full one
@pytest.mark.parametrize("shapes,within", [
    ([(17, 18)], ANY), ([(64, 65)], ANY), ([(100, 101)], ANY), ([(120, 121)], ANY),
    ([(160, 161)], 5000), ([(300, 301)], 4000), ([(400, 400)], 5000), ([(64, 64)] * 3, ANY),
    ([(64, 64)] * 9, ANY), ([(64, 64)] * 30, ANY), ([(125, 125)] * 3, ANY),
    ([(40, 41)] * 40, ANY), ([(172, 172)] * 10, 0), ([(125, 125)] * 19, 0),
    ([(125, 125)] * 20, 0)])
def test_any_numbering_matches_graph_loop(ctx, shapes, within):
    from acousticsim_gb300 import BaraffClothGpu, params
    p = params(max_iters=40, rel_tol=1e-6)
    out = {}
    for solver in ("persistent", "graph_loop"):
        ctx.set_solver(solver)
        cloths = [BaraffClothGpu(ctx, _conf(h, w, "quadratic"), mesh=_mesh(h, w, within))
                  for h, w in shapes]
        for k, c in enumerate(cloths):
            g = np.random.default_rng(70 + k)
            x = c.GetInitPos() + g.normal(0, 2e-4, c.nv * 3)
            c.SetPos(x)
            c.SetPrePos(x - 2e-3 * g.normal(0, 1e-2, c.nv * 3))
        iters = []
        for _ in range(2):
            st = ctx.batch_step(cloths, 0.0, p)
            assert all(s["status"] in ("OK", "MAXITER") and s["solver"] == solver
                       for s in st), st
            iters.append([s["iters"] for s in st])
        out[solver] = iters, [c.GetPos() for c in cloths], [c.get_dx() for c in cloths]
        for c in cloths:
            c.close()
    ctx.set_solver("persistent")
    assert out["persistent"][0] == out["graph_loop"][0]
    for k in (1, 2):
        for a, b in zip(out["persistent"][k], out["graph_loop"][k]):
            assert np.array_equal(a, b)
