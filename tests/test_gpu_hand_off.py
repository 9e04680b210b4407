"""Sets that begin in the graph loop and end in the on-chip kernels: a set of
more cloths than SMs with one that no cluster holds iterates in the graph loop and
hands its last cloths over in the middle of their solves (iteration count, p and
scalars as the loop left them).  The results are those of the loop run to its end,
bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_team import _conf

pytestmark = pytest.mark.gpu

TINY = [(3 + k % 5, 4 + k % 3) for k in range(160)]  # end first
SOFT = [(180, 180)]  # fits no cluster, ends in a few iterations


def _cloths(ctx, tail, others, model):
    from acousticsim_gb300 import BaraffClothGpu
    out = []
    for k, (h, w) in enumerate(tail + others):
        conf = _conf(h, w, model)
        if k >= len(tail) and h > 100:
            conf["cloth_stretch_stiffness"] = [1e-3, 1e-3, 1e-4]
            conf["cloth_bending_stiffness"] = [1e-9, 1e-9]
        c = BaraffClothGpu(ctx, conf)
        g = np.random.default_rng(70 + k)
        x = c.GetInitPos() + g.normal(0, 2e-4, c.nv * 3)
        out.append((c, x, x - 2e-3 * g.normal(0, 1e-2, c.nv * 3)))
    return out


def _step(ctx, cloths, p):
    for c, x, xp in cloths:
        c.Reset()
        c.SetPos(x)
        c.SetPrePos(xp)
    st = ctx.batch_step([c for c, _, _ in cloths], 0.0, p)
    return st, [c.GetPos() for c, _, _ in cloths]


# the cloths that are handed over, and the kernel that ends their solves: a cluster of
# one block and of 16; teams over the GPU with the whole matrix on chip, with the
# stored blocks, with the matrix in memory (up to eight rows a thread and more); more
# rows than such teams hold, in clusters with their stored blocks
@pytest.mark.parametrize("tail,others,model", [
    ([(16, 16)], TINY + SOFT, "quadratic"), ([(64, 64)], TINY + SOFT, "quadratic"),
    ([(64, 64)], TINY + SOFT, "dihedral"), ([(180, 180)], TINY, "quadratic"),
    ([(180, 180)], TINY, "dihedral"), ([(300, 300)], TINY, "quadratic"),
    ([(300, 300)], TINY, "dihedral"), ([(560, 560)], TINY, "quadratic"),
    ([(700, 700)], TINY, "quadratic"), ([(125, 128)] * 24, TINY + SOFT, "quadratic")])
def test_handed_over_solves_are_the_loop_s(built, tail, others, model):
    from acousticsim_gb300 import ClothContext, params
    p = params(max_iters=150, rel_tol=1e-6)
    out = []
    for solver, hand_off in (("graph_loop", 0), ("persistent", 0), ("persistent", len(tail))):
        ctx = ClothContext(0)
        ctx.set_solver(solver)
        ctx.set_tail_hand_off(hand_off)
        cloths = _cloths(ctx, tail, others, model)
        st, x = _step(ctx, cloths, p)
        assert all(s["solver"] == "graph_loop" and s["status"] in ("OK", "MAXITER")
                   for s in st), st
        out.append(([(s["iters"], s["status"]) for s in st], x))
        if hand_off:
            # (the others do end first, and only the on-chip kernels wait for arrivals)
            it = [s["iters"] for s in st]
            assert min(it[:len(tail)]) > max(it[len(tail):]) + 8, it
            ctx.set_spin_limit(1000, 1)
            st, _ = _step(ctx, cloths, p)
            assert [s["status"] for s in st] == ["TIMEOUT"] * len(tail) + ["OK"] * len(others), st
        for c, _, _ in cloths:
            c.close()
        ctx.close()
    for o in out[1:]:
        assert o[0] == out[0][0]
        for a, b in zip(o[1], out[0][1]):
            assert np.array_equal(a, b)
