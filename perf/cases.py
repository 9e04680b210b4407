"""The work a user has this library do, as cases that can be timed and compared.

listed() names the cases, draw() gives more of the same ranges, prepare() makes
what a program holds before the call (cloths, plans, host buffers), run() is
one pass through the public entry points, work() what a pass cannot do
without, and exact() the same results in 64 bits from plain torch and numpy.

Every pass starts from the seeded state (positions are part of the call's
input), so a pass does the same work however often it is repeated.
"""
from __future__ import annotations

import concurrent.futures as cf
import ctypes as C
import functools
import math

import numpy as np
import torch

from acousticsim_gb300 import BaraffClothGpu, ClothContext, params
from acousticsim_gb300 import _native as N
from acousticsim_gb300.cloth import ClothBody, ClothServer

MAX_ITERS = 20000
TOL = 1e-6


# ------------------------------------------------------------------ cases
def listed() -> list[dict]:
    return [
        # a garment patch of an interactive scene: the 20 x 20 cloth at 5 ms, one
        # synchronous step with host buffers; launches and latency count
        {"name": "step_20", "kind": "step", "h": 20, "w": 20, "dt": 5e-3, "k": 1e3},
        # a real-time loop: ten asynchronous warm-started steps, then the positions
        {"name": "frames_64", "kind": "frames", "h": 64, "w": 64, "dt": 2e-3, "k": 1e3,
         "frames": 10},
        # an uneven rectangle with odd sides
        {"name": "step_97x61", "kind": "step", "h": 97, "w": 61, "dt": 2e-3, "k": 1e3},
        # one larger garment, odd sides
        {"name": "step_193x255", "kind": "step", "h": 193, "w": 255, "dt": 2e-3, "k": 1e3},
        # the single large cloth the library is benchmarked on
        {"name": "step_512", "kind": "step", "h": 512, "w": 512, "dt": 2e-3, "k": 1e3},
        # the largest cloth of the benchmarks, at the library's default iteration cap
        {"name": "capped_1024", "kind": "capped", "h": 1024, "w": 1024, "dt": 2e-3, "k": 1e3},
        # a few characters' garments stepped together
        {"name": "batch_12", "kind": "batch", "count": 12, "lo": 16, "hi": 96, "dt": 2e-3},
        # the batched workload: 256 cloths of uneven sizes and stiffness
        {"name": "batch_256", "kind": "batch", "count": 256, "lo": 16, "hi": 128, "dt": 2e-3},
        # a burst of step requests to the request server
        {"name": "serve_48", "kind": "serve", "count": 48, "lo": 16, "hi": 128, "dt": 2e-3},
        # the dihedral-angle bending model (skew block parts in every kernel)
        {"name": "dihedral_128", "kind": "dihedral", "h": 128, "w": 128, "dt": 2e-3, "k": 1e3},
        # contact with a kinematic body
        {"name": "collide_160", "kind": "collide", "h": 160, "w": 160, "dt": 2e-3, "k": 1e3},
        # a stiff step solved to 1e-8 in FP64 by refinement over the FP32 solver
        {"name": "refined_192", "kind": "refined", "h": 192, "w": 192, "dt": 1e-2, "k": 1e4},
    ]


def _logint(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    """One more case: the kinds by how often a program makes the call."""
    kind = rng.choices(["step", "frames", "batch", "serve", "dihedral", "collide", "refined",
                        "capped"], [8, 3, 4, 2, 2, 2, 1, 1])[0]
    if kind == "batch":
        return {"kind": kind, "count": _logint(rng, 3, 240), "lo": rng.randint(12, 40),
                "hi": rng.randint(64, 128), "dt": 2e-3}
    if kind == "serve":
        return {"kind": kind, "count": rng.randint(12, 64), "lo": rng.randint(16, 40),
                "hi": rng.randint(64, 128), "dt": 2e-3}
    top = {"step": 480, "frames": 200, "dihedral": 200, "collide": 224, "refined": 224,
           "capped": 960}[kind]
    low = {"step": 12, "frames": 16, "dihedral": 16, "collide": 64, "refined": 48,
           "capped": 300}[kind]
    h = _logint(rng, low, top)
    w = max(low, min(top, int(h * math.exp(rng.uniform(-0.6, 0.6)))))
    case = {"kind": kind, "h": h, "w": w, "dt": rng.choice([1e-3, 2e-3, 5e-3]),
            "k": rng.choice([3e2, 1e3, 2e3])}
    if kind in ("step", "frames") and h * w > 40000:
        case["dt"], case["k"] = 2e-3, 1e3
    if kind in ("dihedral", "collide", "capped"):
        case["dt"], case["k"] = 2e-3, 1e3
    if kind == "refined":
        case["dt"], case["k"] = 1e-2, rng.choice([1e3, 1e4])
    if kind == "frames":
        case["frames"] = rng.randint(3, 12)
    return case


# ------------------------------------------------------------------ inputs
def _conf(h: int, w: int, k: float, dt: float, model: str = "quadratic", pins: str = "corners"):
    c = {"geometry_type": "regular_triangle", "cloth_size": [1.0, 1.0],
         "subdivision": [h - 1, w - 1], "cloth_init_pos": [0.0, 0.0, 0.0],
         "cloth_uv_rotation": 0, "cloth_stretch_stiffness": [k, k, k / 10],
         "cloth_bending_stiffness": [1e-3, 1e-3], "cloth_density": 0.1,
         "rayleigh_damping_a": 0.01, "rayleigh_damping_b": 0.0, "default_timestep": dt,
         "cloth_bending_model": model}
    if pins == "corners":
        c["constraints"] = {"static_point": [[-0.5, 0.5], [0.5, 0.5]]}
    return c


def _sizes(case: dict) -> list[tuple[int, int, float]]:
    """(h, w, stretch stiffness) of every cloth of a case."""
    if "count" not in case:
        return [(case["h"], case["w"], case["k"])]
    g = np.random.default_rng(7 * case["count"] + 131 * case["lo"] + case["hi"])
    side = np.rint(np.exp(g.uniform(np.log(case["lo"]), np.log(case["hi"]), case["count"])))
    k = np.exp(g.uniform(np.log(1e2), np.log(1e4), case["count"]))
    return [(int(s), int(s), float(x)) for s, x in zip(side, k)]


def _state(case: dict, seed: int) -> tuple[list[np.ndarray], list[np.ndarray]]:
    """x and x_pre of every cloth: the flat rest state with N(0, 1e-3 m) noise
    (a cloth near the dihedral model's or a body's limits: 2e-4 m), velocities
    N(0, 0.01 m/s)."""
    g = np.random.default_rng([seed, 11])
    sx = 2e-4 if case["kind"] in ("dihedral", "collide") else 1e-3
    xs, xps = [], []
    for h, w, _ in _sizes(case):
        p = _rest(h, w)
        x = p + g.normal(0.0, sx, p.shape)
        xs.append(np.ascontiguousarray(x).reshape(-1))
        xps.append((x - case["dt"] * g.normal(0.0, 1e-2, p.shape)).reshape(-1))
    return xs, xps


@functools.lru_cache(maxsize=None)
def _rest(h: int, w: int) -> np.ndarray:
    """Rest positions of the regular grid, vertex i * h + j at column i, row j."""
    i, j = np.meshgrid(np.arange(w), np.arange(h), indexing="ij")
    x = i.reshape(-1) * (1.0 / (w - 1)) - 0.5
    y = j.reshape(-1) * (1.0 / (h - 1)) - 0.5
    return np.stack([x, y, np.zeros_like(x)], 1)


def _sphere(radius=0.25, center=(0.0, -0.05, 0.2515), n_lat=48, n_lon=96):
    """A sphere whose front touches the cloth plane at 1.5 mm."""
    th = np.pi * np.arange(1, n_lat) / n_lat
    ph = 2 * np.pi * np.arange(n_lon) / n_lon
    ring = np.stack([np.outer(np.sin(th), np.cos(ph)), np.outer(np.cos(th), np.ones(n_lon)),
                     np.outer(np.sin(th), np.sin(ph))], -1).reshape(-1, 3)
    c = np.asarray(center)
    pos = c + radius * np.concatenate([[[0.0, 1.0, 0.0]], ring, [[0.0, -1.0, 0.0]]])
    at = lambda a, b: 1 + a * n_lon + b % n_lon  # noqa: E731
    tris = []
    for b in range(n_lon):
        tris += [(0, at(0, b), at(0, b + 1)),
                 (len(pos) - 1, at(n_lat - 2, b + 1), at(n_lat - 2, b))]
        for a in range(n_lat - 2):
            tris += [(at(a, b), at(a + 1, b), at(a + 1, b + 1)),
                     (at(a, b), at(a + 1, b + 1), at(a, b + 1))]
    tris = np.array(tris, np.int32)
    v0, v1, v2 = pos[tris[:, 0]], pos[tris[:, 1]], pos[tris[:, 2]]
    inward = np.einsum("ij,ij->i", np.cross(v1 - v0, v2 - v1), v0 + v1 + v2 - 3 * c) <= 0
    tris[inward] = tris[inward][:, [0, 2, 1]]
    return pos, tris


def _pinned(n: int) -> np.ndarray:
    """Host buffer a program exchanges positions through (page-locked)."""
    t = torch.empty(n, dtype=torch.float64)
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


# ------------------------------------------------------------------ prepare
def prepare(case: dict, seed: int) -> dict:
    kind, dt = case["kind"], case["dt"]
    ctx = ClothContext(0)
    pins = "edge" if "count" in case else "corners"
    model = "dihedral" if kind == "dihedral" else "quadratic"

    def make(s):
        h, w, k = s
        c = BaraffClothGpu(ctx, _conf(h, w, k, dt, model, pins))
        if pins == "edge":
            c.AddConstraintStaticVertices([i * h + h - 1 for i in range(w)])
        return c

    sizes = _sizes(case)
    if len(sizes) > 1:
        with cf.ThreadPoolExecutor(8) as ex:
            cloths = list(ex.map(make, sizes))
    else:
        cloths = [make(sizes[0])]
    xs, xps = _state(case, seed)
    total = sum(x.size for x in xs)
    bx, bp, bo = _pinned(total), _pinned(total), _pinned(total)
    cut = np.cumsum([0] + [x.size for x in xs])
    views = []
    for i, (x, xp) in enumerate(zip(xs, xps)):
        a, b = cut[i], cut[i + 1]
        bx[a:b], bp[a:b] = x, xp
        views.append((bx[a:b], bp[a:b], bo[a:b]))
    s = {"kind": kind, "dt": dt, "ctx": ctx, "cloths": cloths, "views": views, "out": bo,
         "frames": case.get("frames", 0),
         "p": params(max_iters=MAX_ITERS, rel_tol=TOL, warm_start=(kind == "frames"))}
    if kind == "capped":
        s["p"] = params(max_iters=1000, rel_tol=TOL, warm_start=False)
    if kind == "collide":
        s["body"] = ClothBody(ctx, *_sphere())
        cloths[0].set_bodies([s["body"]])
    if kind == "refined":
        s["p"] = params(max_iters=6000, rel_tol=1e-5, warm_start=False)
        cloths[0].SetPos(views[0][0])
        cloths[0].SetPrePos(views[0][1])
    if kind == "serve":
        srv = ClothServer(ctx, 40 << 30, 0, 16)
        for c in cloths:
            srv.add(c, dt, s["p"])
        srv.start()
        s["server"] = srv
    return s


# ------------------------------------------------------------------ run
def run(s: dict):
    kind, cloths, views = s["kind"], s["cloths"], s["views"]
    if kind in ("step", "capped", "dihedral", "collide"):
        x, xp, out = views[0]
        st = cloths[0].step_host(x, xp, out, s["dt"], s["p"])
        return {"x": out, "iters": st["iters"]}
    if kind == "frames":
        c = cloths[0]
        c.Reset()  # the warm start of the first frame
        c.SetPos(views[0][0])
        c.SetPrePos(views[0][1])
        for _ in range(s["frames"]):
            c.step_async(s["dt"], s["p"])
        _get_pos(c, views[0][2])
        return {"x": s["out"]}
    if kind == "refined":
        cloths[0].assemble(s["dt"])
        st = cloths[0].solve_refined(s["p"], 1e-8, 20)
        return {"dx": cloths[0].get_dx(), "outer": st["outer"], "inner": st["inner_iters"]}
    for c, (x, xp, _) in zip(cloths, views):
        c.SetPos(x)
        c.SetPrePos(xp)
    if kind == "batch":
        iters = [st["iters"] for st in s["ctx"].batch_step(cloths, s["dt"], s["p"])]
    else:
        srv = s["server"]
        for i in range(len(cloths)):
            srv.submit(i, i)
        iters, left = [0] * len(cloths), len(cloths)
        while left:
            for r in srv.poll(wait_s=0.05):
                iters[r["tag"]] = r["iters"]
                left -= 1
    for c, (_, _, out) in zip(cloths, views):
        _get_pos(c, out)
    return {"x": s["out"], "iters": np.array(iters, np.int64)}


def _get_pos(c: BaraffClothGpu, out: np.ndarray) -> None:
    """cloth_get_pos into the program's own buffer."""
    N.call("cloth_get_pos", c.handle, N.ptr(out, C.c_double), c.nv)


# ------------------------------------------------------------------ work
def work(case: dict) -> dict:
    """Bytes: x, x_pre and x (FP64), the mesh and the assembled system once.
    Flops: assembly, and PCG iterations of a block-Jacobi PCG (about 11 blocks
    a row); their number grows with the grid and with dt sqrt(k)."""
    nbytes = flops = 0.0
    for h, w, k in _sizes(case):
        nv, side = h * w, max(h, w)
        stiff = case["dt"] * math.sqrt(k / 0.1)  # metres a wave travels in a step
        iters = min(MAX_ITERS, 20 + 2.2 * side * min(1.0, stiff * 2) * math.sqrt(max(1, side / 128)))
        if case["kind"] == "capped":
            iters = 1000
        if case["kind"] == "refined":
            iters *= 4
        steps = case.get("frames", 1)
        nbytes += nv * (72.0 + 2 * 76 + 11 * 36 * steps)
        flops += steps * nv * (1200.0 + iters * (11 * 18 + 40))
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ 64 bits
def _grid(h: int, w: int):
    """Material coordinates (float), triangles, and interior edge stencils
    (two edge vertices, two opposite ones, their triangles) of the grid."""
    p = _rest(h, w)
    uv = p[:, :2].astype(np.float32)
    col, row = np.meshgrid(np.arange(h - 1), np.arange(w - 1))
    lu = (row * h + col).reshape(-1)
    even = ((row + col) % 2 == 0).reshape(-1, 1)
    ru, ld, rd = lu + 1, lu + h, lu + h + 1
    t1 = np.where(even, np.stack([lu, ld, rd], 1), np.stack([lu, ld, ru], 1))
    t2 = np.where(even, np.stack([lu, rd, ru], 1), np.stack([ld, rd, ru], 1))
    tris = np.stack([t1, t2], 1).reshape(-1, 3)
    e = np.concatenate([tris[:, [0, 1, 2]], tris[:, [1, 2, 0]], tris[:, [2, 0, 1]]])
    tri = np.tile(np.arange(len(tris)), 3)
    key = np.minimum(e[:, 0], e[:, 1]).astype(np.int64) * len(p) + np.maximum(e[:, 0], e[:, 1])
    o = np.argsort(key, kind="stable")
    at = np.flatnonzero(key[o][1:] == key[o][:-1])
    a, b = o[at], o[at + 1]
    st = np.stack([e[a, 0], e[a, 1], e[a, 2], e[b, 2]], 1)
    return p, uv, tris, st, np.stack([tri[a], tri[b]], 1)


class _Exact:
    """The cloths of a case as one mesh without shared vertices, in FP64."""

    def __init__(self, case: dict, seed: int):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        f32 = lambda v: float(np.float32(v))  # noqa: E731  parameters the library holds as float
        dih = case["kind"] == "dihedral"
        P, UV, T, S, ST, K, PIN = [], [], [], [], [], [], []
        nv = nt = 0
        for h, w, k in _sizes(case):
            p, uv, tris, st, stt = _grid(h, w)
            P.append(p)
            UV.append(uv)
            T.append(tris + nv)
            S.append(st + nv)
            ST.append(stt + nt)
            K.append(np.tile([[f32(k), f32(k), f32(k / 10)]], (len(tris), 1)))
            top = nv + np.arange(w) * h + h - 1
            PIN.append(top if "count" in case else top[[0, -1]])
            nv, nt = nv + len(p), nt + len(tris)
        t = lambda a, d=torch.float64: torch.as_tensor(np.concatenate(a), dtype=d, device=self.dev)  # noqa: E731
        self.nv, self.rest, uv = nv, t(P), t(UV)
        self.tris, self.st, stt = t(T, torch.int64), t(S, torch.int64), t(ST, torch.int64)
        self.ks, self.pins = t(K), t(PIN, torch.int64)
        self.dt = f32(case["dt"])
        p, tr = self.rest, self.tris
        area = 0.5 * torch.linalg.norm(torch.linalg.cross(p[tr[:, 1]] - p[tr[:, 0]],
                                                          p[tr[:, 2]] - p[tr[:, 0]]), dim=1)
        self.area = area
        m = torch.zeros(nv, dtype=torch.float64, device=self.dev)
        for a in range(3):
            m.index_add_(0, tr[:, a], area / 3 * f32(0.1))
        self.m = m
        # stretch coefficients: Dm^-1, and Dm^-1 in the frame turned by 45 degrees
        D = torch.stack([uv[tr[:, 1]] - uv[tr[:, 0]], uv[tr[:, 2]] - uv[tr[:, 0]]], 2)
        Di = torch.linalg.inv(D)
        r = math.sqrt(0.5)
        R = torch.tensor([[r, r], [-r, r]], dtype=torch.float64, device=self.dev)
        self.coef = []
        for M in (Di, Di @ R):
            c = [torch.stack([-M[:, 0, q] - M[:, 1, q], M[:, 0, q], M[:, 1, q]], 1) for q in (0, 1)]
            self.coef.append(c)
        s = self.st
        if dih:
            ln = lambda a, b: torch.linalg.norm(p[a] - p[b], dim=1)  # noqa: E731
            le = ln(s[:, 0], s[:, 1])
            hs = 2 * (area[stt[:, 0]] + area[stt[:, 1]]) / le
            self.dfac = -f32(1e-3) * le / hs
        else:
            cot = lambda a, b, c: self._cot(p[a], p[b], p[c])  # noqa: E731
            c1, c2 = cot(s[:, 0], s[:, 1], s[:, 2]), cot(s[:, 0], s[:, 1], s[:, 3])
            c3, c4 = cot(s[:, 1], s[:, 0], s[:, 2]), cot(s[:, 1], s[:, 0], s[:, 3])
            v = torch.stack([c3 + c4, c1 + c2, -c1 - c3, -c2 - c4], 1)
            pre = 3.0 / (area[stt[:, 0]] + area[stt[:, 1]])
            self.qb = v[:, :, None] * v[:, None, :] * (pre * f32(1e-3))[:, None, None]
        self.dihedral = dih
        xs, xps = _state(case, seed)
        put = lambda v: torch.as_tensor(np.concatenate(v), device=self.dev).reshape(-1, 3)  # noqa: E731
        self.x, self.xp = put(xs), put(xps)

    @staticmethod
    def _cot(a, b, c):
        u, v = b - a, c - a
        d = (u * v).sum(1)
        return d / torch.sqrt((u * u).sum(1) * (v * v).sum(1) - d * d)

    def system(self):
        """A (sparse) and b of the implicit step from x, x_pre."""
        nv, tr, x = self.nv, self.tris, self.x
        I3 = torch.eye(3, dtype=torch.float64, device=self.dev)
        f = torch.zeros(nv, 3, dtype=torch.float64, device=self.dev)
        f[:, 1] = -9.8 * self.m
        rows, cols, vals = [], [], []

        def add(i, j, B):
            rows.append(i)
            cols.append(j)
            vals.append(B)

        for q, (cu, cv) in enumerate(self.coef):
            Ku, Kv = (self.ks[:, 0], self.ks[:, 1]) if q == 0 else (self.ks[:, 2], self.ks[:, 2])
            X = x[tr]
            Fu, Fv = (cu[:, :, None] * X).sum(1), (cv[:, :, None] * X).sum(1)
            nu, nw = torch.linalg.norm(Fu, dim=1), torch.linalg.norm(Fv, dim=1)
            u, v = Fu / nu[:, None], Fv / nw[:, None]
            D = []
            for n in (u, v):  # both terms divide by |Fu|
                D.append(n[:, :, None] * n[:, None, :] / nu[:, None, None]
                         + torch.clamp(1 - 1 / nu, min=0)[:, None, None] * I3)
            for a in range(3):
                f.index_add_(0, tr[:, a], -(self.area * Ku * (nu - 1) * cu[:, a])[:, None] * u
                             - (self.area * Kv * (nw - 1) * cv[:, a])[:, None] * v)
                for b in range(3):
                    add(tr[:, a], tr[:, b],
                        -(self.area * Ku * cu[:, a] * cu[:, b])[:, None, None] * D[0]
                        - (self.area * Kv * cv[:, a] * cv[:, b])[:, None, None] * D[1])
        s = self.st
        if self.dihedral:
            v0, v1, v2, v3 = (x[s[:, a]] for a in range(4))
            cr = lambda a, b: torch.linalg.cross(a, b)  # noqa: E731
            dot = lambda a, b: (a * b).sum(1, keepdim=True)  # noqa: E731
            e = v1 - v0
            n0, n1 = cr(e, v2 - v1), cr(v0 - v1, v3 - v0)
            le = torch.sqrt(dot(e, e))
            h0, h1 = n0 / torch.sqrt(dot(n0, n0)), n1 / torch.sqrt(dot(n1, n1))
            beta = torch.atan2(dot(e / le, cr(h0, h1)), dot(h0, h1))
            g0, g1 = -cr(e, n0) / (le * dot(n0, n0)), cr(e, n1) / (le * dot(n1, n1))
            G = [cr(v1 - v2, g0) + cr(v3 - v1, g1), cr(v2 - v0, g0) + cr(v0 - v3, g1),
                 cr(v0 - v1, g0), cr(v1 - v0, g1)]
            c = self.dfac[:, None]
            for a in range(4):
                f.index_add_(0, s[:, a], c * beta / 2 * G[a])
                for b in range(4):
                    add(s[:, a], s[:, b], c[:, :, None] * G[a][:, :, None] * G[b][:, None, :])
        else:
            for a in range(4):
                for b in range(4):
                    f.index_add_(0, s[:, a], -self.qb[:, a, b, None] * x[s[:, b]])
                    add(s[:, a], s[:, b], -self.qb[:, a, b, None, None] * I3)
        h = self.dt
        fixed = torch.zeros(nv, dtype=torch.bool, device=self.dev)
        fixed[self.pins] = True
        i, j, B = torch.cat(rows), torch.cat(cols), torch.cat(vals)
        on = (i == j) | ~(fixed[i] | fixed[j])
        i, j, B = i[on], j[on], -h * h * B[on]
        d = torch.arange(nv, device=self.dev)
        i, j = torch.cat([i, d]), torch.cat([j, d])
        B = torch.cat([B, ((1 + h * float(np.float32(0.01))) * self.m)[:, None, None] * I3])
        k = torch.arange(3, device=self.dev)
        ij = torch.stack([(3 * i[:, None, None] + k[None, :, None]).expand_as(B).reshape(-1),
                          (3 * j[:, None, None] + k[None, None, :]).expand_as(B).reshape(-1)])
        A = torch.sparse_coo_tensor(ij, B.reshape(-1), (3 * nv, 3 * nv)).coalesce()
        M = torch.zeros(nv, 3, 3, dtype=torch.float64, device=self.dev)
        M.index_add_(0, i[i == j], B[i == j])
        b = h * h * f + self.m[:, None] * (self.x - self.xp)
        b[fixed] = 0
        return A.to_sparse_csr(), torch.linalg.inv(M), b

    def solve(self, tol: float = 1e-11, most: int = 40000):
        """dx of A dx = b by PCG in 64 bits."""
        A, M, b = self.system()
        mul = lambda v: (A @ v.reshape(-1, 1)).reshape(-1, 3)  # noqa: E731
        pre = lambda r: (M @ r[:, :, None])[:, :, 0]  # noqa: E731
        x, r = torch.zeros_like(b), b.clone()
        z = pre(r)
        p, rz, stop = z.clone(), (r * z).sum(), tol * float(torch.linalg.norm(b))
        for it in range(most):
            q = mul(p)
            a = rz / (p * q).sum()
            x += a * p
            r -= a * q
            if it % 50 == 49 and float(torch.linalg.norm(r)) <= stop:
                break
            z = pre(r)
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
        return x

    def step(self):
        tgt = self.rest[self.pins].to(torch.float32).to(torch.float64)
        self.x[self.pins] = tgt
        self.xp[self.pins] = tgt
        dx = self.solve()
        self.xp = self.x.clone()
        self.x = self.x + dx
        return dx


def exact(case: dict, seed: int):
    """run()'s outputs in 64 bits; nothing for contacts and for a solve that the
    iteration cap ends (the value depends on the iteration, not on the system)."""
    if case["kind"] in ("collide", "capped"):
        return None
    e = _Exact(case, seed)
    if case["kind"] == "refined":
        tgt = e.rest[e.pins].to(torch.float32).to(torch.float64)
        e.x[e.pins] = tgt
        e.xp[e.pins] = tgt
        return {"dx": e.solve().reshape(-1).cpu().numpy(), "outer": None, "inner": None}
    for _ in range(case.get("frames", 1)):
        e.step()
    return {"x": e.x.reshape(-1).cpu().numpy(), "iters": None}
