"""The on-chip persistent PCG (k_pcg_team) against the graph loop, the other
driver of the same arithmetic: iterations and positions agree bit for bit (row
operations are the same code in the same order, sums above 32 rows are exact),
at the edges of its row split."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _conf(h, w, model):
    return {"geometry_type": "regular_triangle", "cloth_size": [1.0, 1.0],
            "subdivision": [h - 1, w - 1], "cloth_init_pos": [0.0, 0.0, 0.0],
            "cloth_uv_rotation": 0, "cloth_stretch_stiffness": [1e3, 1e3, 1e2],
            "cloth_bending_stiffness": [1e-3, 1e-3], "cloth_density": 0.1,
            "rayleigh_damping_a": 0.01, "rayleigh_damping_b": 0.0, "default_timestep": 2e-3,
            "cloth_bending_model": model,
            "constraints": {"static_point": [[-0.5, 0.5], [0.5, 0.5]]}}


# one row short of, at and past a 32-row chunk; around the most rows of one
# row per thread in a single block (480); the largest single
# block and the smallest team; a short last block; a set whose teams hold two
# rows per thread; uneven teams in one launch; sets of cloths too large for the
# whole matrix on chip: every stored block on chip, and a part of them (with
# rows whose transposed blocks another block owns), two, three and four rows a
# thread; the matrix in memory, up to eight rows a thread and more; a set of
# those; more cloths than SMs, of every size of cluster, the largest with their stored
# blocks alone
MANY = [(3 + k % 5, 4 + k % 3) for k in range(160)] + [(22, 23), (30, 33), (44, 45), (62, 61),
                                                       (87, 88), (100, 100), (125, 128)]


@pytest.mark.parametrize("model", ["quadratic", "dihedral"])
@pytest.mark.parametrize("shapes", [[(2, 2)], [(3, 7)], [(4, 8)],
                                    [(3, 11)], [(16, 32)], [(19, 27)], [(20, 32)], [(21, 31)],
                                    [(65, 64)], [(128, 129)],
                                    [(150, 150), (149, 150), (150, 149), (140, 150)],
                                    [(5, 5), (90, 31), (2, 40), (64, 64)], [(270, 300)],
                                    [(300, 320), (5, 5)], [(400, 401)], [(470, 480)], [(541, 560)],
                                    [(610, 650)], [(760, 767)], [(771, 770)], [(520, 530), (9, 7), (350, 360)], MANY])
def test_team_kernel_matches_graph_loop(ctx, shapes, model):
    from acousticsim_gb300 import BaraffClothGpu, params
    big = sum(h * w for h, w in shapes) > 40000  # a few iterations show it
    p = params(max_iters=60 if big else 4000, rel_tol=1e-6)
    out = {}
    for solver in ("persistent", "graph_loop"):
        ctx.set_solver(solver)
        cloths = [BaraffClothGpu(ctx, _conf(h, w, model)) for h, w in shapes]
        for k, c in enumerate(cloths):
            g = np.random.default_rng(70 + k)
            x = c.GetInitPos() + g.normal(0, 2e-4, c.nv * 3)
            c.SetPos(x)
            c.SetPrePos(x - 2e-3 * g.normal(0, 1e-2, c.nv * 3))
        iters = []
        for _ in range(2):  # the second step starts from the first one's dx
            st = ctx.batch_step(cloths, 0.0, p)
            assert all(s["status"] in (("OK", "MAXITER") if big else ("OK",)) and
                       s["solver"] == solver for s in st), st
            iters.append([s["iters"] for s in st])
        out[solver] = iters, [c.GetPos() for c in cloths], [c.get_dx() for c in cloths]
        for c in cloths:
            c.close()
    ctx.set_solver("persistent")
    assert out["persistent"][0] == out["graph_loop"][0]
    for k in (1, 2):
        for a, b in zip(out["persistent"][k], out["graph_loop"][k]):
            assert np.array_equal(a, b)
