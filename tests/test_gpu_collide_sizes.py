"""Contacts, contact Hessian and repulsion against the FP64 oracle where the
device's collision kernels change their way: more hits on one edge or point than
a warp keeps, longer contact lists than it ranks, and more contacts than the
repulsion stages, lists or counts in shared memory."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


def _patch(n, h, centre):
    """A slightly wavy grid of n x n cells of h, 1 mm under the plane z = centre z,
    turned so that none of its edges is parallel to the cloth's (the normal of two
    parallel edges is 0 / 0)."""
    i = np.arange(n + 1)
    a, b = np.meshgrid(i, i, indexing="ij")
    c, s = np.cos(0.3), np.sin(0.3)
    u, v = (a - n / 2) * h, (b - n / 2) * h
    pos = np.stack([centre[0] + c * u - s * v, centre[1] + s * u + c * v,
                    centre[2] - 1e-3 + 4e-4 * np.sin(1.3 * a) * np.cos(0.7 * b)], -1)
    q = (i[:-1, None] * (n + 1) + i[None, :-1]).reshape(-1)
    t = np.concatenate([np.stack([q, q + 1, q + n + 1], -1),
                        np.stack([q + 1, q + n + 2, q + n + 1], -1)])
    return pos.reshape(-1, 3), np.ascontiguousarray(t, np.int32)


# cloth cells, body cells, body cell size: a few contacts; hundreds; an edge with
# more hits than are kept and rows whose Hessian records do not fit; a fine cloth
# whose contacts are more than are staged; more than there are counts for
@pytest.mark.parametrize("sub,n,h", [(5, 1, 0.02), (5, 14, 0.002), (5, 30, 0.0015), (40, 6, 0.02),
                                     (70, 24, 0.005)])
def test_collision_sizes(ctx, built, sub, n, h):
    from acousticsim_gb300 import BaraffClothGpu, ClothBody, params
    from oracle import oracle as orc
    dt = 2e-3
    conf = {"geometry_type": "regular_triangle", "cloth_size": [0.15, 0.15],
            "subdivision": [sub, sub], "cloth_init_pos": [0.0, 0.0, 0.0],
            "cloth_uv_rotation": 0, "cloth_stretch_stiffness": [1e3, 1e3, 1e2],
            "cloth_bending_stiffness": [1e-3, 1e-3], "cloth_density": 0.1,
            "rayleigh_damping_a": 0.01, "rayleigh_damping_b": 0.0, "default_timestep": dt}
    cl = BaraffClothGpu(ctx, conf)
    x = cl.GetPos().copy()
    p = x.reshape(-1, 3)
    assert np.ptp(p[:, 2]) == 0
    pos, tris = _patch(n, h, (p.min(0) + p.max(0)) / 2 + [4e-3, -3e-3, 0])
    body = ClothBody(ctx, pos.reshape(-1), tris.reshape(-1))
    tn, vn = orc.body_normals(pos, tris)
    ref = orc.contacts(cl.mesh, x, {"pos": pos, "tris": tris, "edges": orc.derive_edges(tris),
                                    "tnormal": tn, "vnormal": vn})
    tab = orc.tables(cl.mesh, 0.1, [1e-3, 1e-3])
    cl.SetPos(x)
    cl.SetPrePos(x + np.tile([0.0, 0.0, 1e-4], x.size // 3))
    cl.assemble()
    without = cl.export_system()["A"].astype(np.float64)
    cl.set_bodies([body])
    # (the default pair list, sized by the cloth, holds all but the last case's)
    cl.set_contact_capacity(1 << 20 if sub == 70 else 0, len(ref["pt_i"]) + 8,
                            len(ref["ee_i"]) + 8)
    cl.assemble()
    con = cl.get_contacts()
    print(sub, n, h, "contacts", len(con["pt_i"]), len(con["ee_i"]))
    assert con["overflow"] == 0
    assert np.array_equal(con["pt_i"], ref["pt_i"])
    assert np.array_equal(con["ee_i"], ref["ee_i"])
    # the bounds of the reference's own contact lists
    assert np.abs(con["pt_d"] - ref["pt_d"]).max() < 1e-15
    assert np.abs(con["ee_d"] - ref["ee_d"]).max() < 1e-15
    # the matrix entries are FP32, the Hessian is the difference of two, and up to
    # ~1,000 contacts of a vertex are summed in FP32 (each rounding 2^-24)
    H = cl.export_system()["A"].astype(np.float64) - without
    want = orc.contact_hessian(tab, cl.mesh, ref)
    eps = np.abs(without).max() * 2.0 ** -23
    assert np.abs(H - want).max() <= eps + 1e-4 * np.abs(want).max()

    st = cl.UpdatePos(0.0, params(max_iters=20000, rel_tol=1e-6))
    assert st["status"] == "OK", st
    con = cl.get_contacts()
    dx, dxr = cl.get_dx(), cl.get_repulsed_dx()
    out = orc.repulsion(cl.mesh, tab["mass"], conf["cloth_stretch_stiffness"], dt, con, dx)
    assert np.abs(out - dx).max() > 0
    err = rel(dxr - dx, out - dx)
    print("repulsion rounds", con["repulsion_rounds"], "error", err)
    assert err < 1e-12
    cl.set_bodies([])
    cl.close()
    body.close()
