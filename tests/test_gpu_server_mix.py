"""Requests of all sizes in one server: cloths that fit a thread-block cluster
iterate in the on-chip kernels, larger ones beside them in the graph loop, over
several chunks; every result is that of the cloth stepped alone, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import test_server as T

pytestmark = pytest.mark.gpu

# (side, stiffness, steps): clusters of one block, of several, of 16 with the whole
# matrix, with the stored blocks and with a part of them; past 30,720 rows the graph loop
WORK = [(12, 3e2, 3), (180, 3e2, 2), (40, 1e3, 2), (64, 3e2, 2), (190, 1e2, 1), (100, 3e2, 2),
        (126, 1e2, 1), (160, 1e2, 1)]
IN_LOOP = [side * side > 30720 for side, _, _ in WORK]


@pytest.mark.parametrize("chunk_iters", [8, 50])
def test_loop_and_clusters_side_by_side(ctx, chunk_iters):
    from acousticsim_gb300 import params
    p = params(max_iters=5000, rel_tol=T.REL_TOL)
    alone = T._twins(ctx, WORK, p)
    served, stats = T._serve(ctx, WORK, p, budget=4 << 30, max_inflight=0,
                             chunk_iters=chunk_iters)
    assert stats["max_inflight_seen"] > 2
    T._check_same(served, alone)


def test_which_requests_wait_for_arrivals(built):
    """Which of them the on-chip kernels ran: those whose bounded waits run out."""
    from acousticsim_gb300 import ClothContext, ClothServer, params
    ctx = ClothContext(0)
    srv = ClothServer(ctx, 4 << 30, 0, 8)
    cloths = [T._cloth(ctx, n, k, 100 + i) for i, (n, k, _) in enumerate(WORK)]
    for c in cloths:
        srv.add(c, 0.0, params(max_iters=5000, rel_tol=T.REL_TOL))
    srv.start()
    ctx.set_spin_limit(1000, 1)
    for i in range(len(WORK)):
        srv.submit(i, i)
    srv.drain(60.0)
    res = {r["tag"]: r["status"] for r in srv.poll()}
    assert [res[i] for i in range(len(WORK))] == ["OK" if q else "TIMEOUT" for q in IN_LOOP], res
    srv.close()
    for c in cloths:
        c.close()
    ctx.close()
