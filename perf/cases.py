"""The workloads the framework is timed on, and their values in 64 bits.

Every case is work a program hands to the public classes (Cloth, Batch, Server,
SoftBody): it restores a snapshot of the simulation, advances it some frames
and reads the state back -- what rollback, look-ahead and replay loops do, and
what makes one pass the same work as the next.  The snapshots are synthetic:
sheets waved or draped without stretching beyond a few tenths of a percent,
blocks bent by a few percent, both moving, so that forces, contacts and the
CG's iteration counts are those of a running simulation.

Kinds:
  cloth     one cloth (grid or two sewn panels), any solver option and CG
            strategy, optionally draped over a sphere or a rod
  batch     many cloths of uneven sizes, stepped together
  server    requests submitted to the continuous-batching server and drained
  softbody  a tetrahedral block hanging from one node
  self      a folded cloth with particle-triangle contacts (thickness > 0)
"""
import math

import numpy as np
import torch

import bounce_b200 as b3g

DT = 1.0 / 60.0
GRAVITY = (0.0, -9.8, 0.0)
EXTENSION, SLOP, BAUMGARTE, MAX_CORRECTION = 0.2, 0.005, 0.1, 0.2  # the step's contact constants


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def _cloth(name, side, shape="grid", bending=0.0, stretch=1e4, shear=1e3, damping=0.05, collider="none",
           stop="relative", dot="f64", limit=200, cg="persistent", frames=4):
    return {"name": name, "kind": "cloth", "shape": shape, "side": side, "bending": bending, "stretch": stretch,
            "shear": shear, "damping": damping, "collider": collider, "stop": stop, "dot": dot, "limit": limit,
            "cg": cg, "frames": frames}


def listed():
    return [
        # a handkerchief-sized cloth in a game: one frame at a time with every default; latency is all of it
        _cloth("tiny_grid8", 8, stop="reference", dot="f32", limit=20, cg="launches", frames=1),
        # the plain method's cloth: 1,024 vertices, CG to 1e-4 with at most 50 iterations
        _cloth("plain_grid32", 32, limit=50, cg="launches"),
        # a garment part: two panels sewn along their edges, default strategy and stop rule
        _cloth("sewn_panels45", 45, shape="sewn", stop="reference", dot="f32", limit=20, cg="launches"),
        # an odd-sized curtain over a rod with bending springs, the reference's 20-iteration rule
        _cloth("rod_grid91", 91, bending=1e2, collider="rod", stop="reference", dot="f32", limit=20),
        # the headline cloth: 65,536 vertices, bending, draped over a sphere, CG to 1e-4
        _cloth("sphere_grid256", 256, bending=1e2, collider="sphere"),
        # a large garment in the one-reduction form, odd side
        _cloth("fused_grid383", 383, cg="fused", stop="relative", dot="f64", limit=200, frames=2),
        # the ill-conditioned million-vertex cloth, in the form that is used there
        _cloth("stiff_grid1024", 1024, stretch=1e5, damping=0.1, cg="fused", limit=2000, frames=6),
        # many cloths of uneven sizes at once (a crowd, or a data-generation job)
        {"name": "batch128", "kind": "batch", "count": 128, "lo": 16, "hi": 128, "frames": 16, "limit": 50},
        # a burst of requests to the step server, a quarter of them over a sphere
        {"name": "server40", "kind": "server", "requests": 40, "lo": 8, "hi": 96, "most": 12},
        # the large block: 68,921 nodes, 320,000 tetrahedra
        {"name": "block40", "kind": "softbody", "w": 40, "h": 40, "d": 40, "plastic": False, "frames": 4,
         "cg": "persistent"},
        # a jelly in a game, of a material that yields, frame by frame
        {"name": "jelly7", "kind": "softbody", "w": 7, "h": 7, "d": 7, "plastic": True, "frames": 1,
         "cg": "persistent"},
        # a sheet folded onto itself
        {"name": "folded24", "kind": "self", "side": 24, "gap": 0.37, "frames": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cloth", "cloth", "cloth", "cloth", "batch", "server", "softbody", "softbody", "self"])
    if kind == "batch":
        lo = _log(rng, 8, 40)
        return {"kind": "batch", "count": _log(rng, 8, 120), "lo": lo, "hi": rng.randint(lo + 8, 128),
                "frames": rng.randint(4, 16), "limit": rng.choice([20, 50, 200])}
    if kind == "server":
        lo = _log(rng, 8, 24)
        return {"kind": "server", "requests": _log(rng, 6, 40), "lo": lo, "hi": rng.randint(lo + 4, 96),
                "most": rng.randint(2, 12)}
    if kind == "softbody":
        plastic = rng.random() < 0.3
        return {"kind": "softbody", "w": _log(rng, 3, 40), "h": _log(rng, 3, 40), "d": _log(rng, 3, 39),
                "plastic": plastic, "frames": 1 if plastic else rng.randint(1, 4), "cg": rng.choice(["persistent", "persistent", "fused", "launches"])}
    if kind == "self":
        return {"kind": "self", "side": _log(rng, 8, 28), "gap": rng.uniform(0.35, 0.39), "frames": rng.randint(2, 3)}
    shape = rng.choice(["grid", "grid", "grid", "sewn"])
    side = _log(rng, 8, 700 if shape == "grid" else 160)
    collider = rng.choice(["none", "sphere", "rod"]) if shape == "grid" and side <= 400 else "none"
    stop, dot, limit = rng.choice([("reference", "f32", 20), ("relative", "f64", 50), ("relative", "f64", 200)])
    cg = rng.choice(["persistent", "persistent", "fused"] + (["launches"] if side <= 128 else []))
    c = _cloth("", side, shape=shape, bending=rng.choice([0.0, 1e2]), stretch=10.0 ** rng.uniform(3.5, 5.0),
               shear=10.0 ** rng.uniform(2.5, 3.5), damping=rng.choice([0.05, 0.1]), collider=collider, stop=stop,
               dot=dot, limit=limit, cg=cg, frames=rng.randint(1, 4))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _jitter(side):
    return min(1e-3, 0.25 / (side - 1)) if side <= 512 else 0.0


def _options(stop, dot, limit):
    if stop == "reference":
        return b3g.SolverOptions(b3g.STOP_REFERENCE, 0.0, limit, {"f32": b3g.DOT_F32, "f64": b3g.DOT_F64}[dot])
    return b3g.SolverOptions.relative(1e-4, limit, {"f32": b3g.DOT_F32, "f64": b3g.DOT_F64}[dot])


def _curve(u, turn):
    """The point at arc length u of a plane curve whose direction is turn(u)."""
    s = np.linspace(u.min(), u.max(), 4096)
    a = turn(s)
    step = s[1] - s[0]
    x = np.concatenate([[0.0], np.cumsum(0.5 * step * (np.cos(a[1:]) + np.cos(a[:-1])))])
    y = np.concatenate([[0.0], np.cumsum(0.5 * step * (np.sin(a[1:]) + np.sin(a[:-1])))])
    zero = np.argmin(np.abs(s))
    return np.interp(u, s, x - x[zero]), np.interp(u, s, y - y[zero])


def _snapshot(vertices, pinned, rng, collider):
    """A bent and moving sheet: x, v and the last step's velocity change."""
    u, h, w = (vertices[:, k].astype(np.float64) for k in range(3))
    if collider == "none":
        amount, phase, waves = rng.uniform(0.3, 0.5), rng.uniform(0.0, 6.28), rng.uniform(1.0, 2.0)
        px, py = _curve(u, lambda s: amount * np.sin(6.28 * waves * s + phase))
    else:
        radius, top = (0.2995, -0.2) if collider == "sphere" else (0.0995, -0.3)
        lean = rng.uniform(0.4, 0.7)
        reach = lean * radius
        px, py = _curve(u, lambda s: -np.clip(s, -reach, reach) / radius)
        py = py + (top + (radius - (0.3 if collider == "sphere" else 0.1)))
    x = np.stack([1.002 * px, py + h, 1.002 * w], 1)
    speed = rng.uniform(0.3, 0.8)
    v = np.zeros_like(x)
    v[:, 0] = 0.1 * speed * np.cos(5.0 * w + 3.0 * u)
    v[:, 1] = -speed * (0.6 + 0.4 * np.cos(4.0 * u) * np.cos(3.0 * w))
    v[:, 2] = 0.1 * speed * np.sin(4.0 * u)
    v += rng.normal(0.0, 1e-3, v.shape)
    v[pinned] = 0.0
    return x.astype(np.float32), v.astype(np.float32), np.zeros(x.shape, np.float32)


def _cloth_scene(case, seed):
    side, rng = int(case["side"]), np.random.default_rng(seed)
    if case["shape"] == "sewn":
        scene = b3g.sewn_scene(side, seed=seed % 1000003)
    else:
        mesh = b3g.grid_mesh(side, 1.0, _jitter(side), seed)
        pins = np.array([0, side - 1], np.uint32)
        scene = b3g.Scene("sheet", mesh, b3g.ClothDef(density=1.0, friction=0.3), pins, gravity=GRAVITY)
        if case["collider"] == "sphere":
            scene.spheres = [((0.0, -0.5, 0.0), 0.3, 0.3)]
        elif case["collider"] == "rod":
            scene.capsules = [((0.0, -0.4, -0.6), (0.0, -0.4, 0.6), 0.1, 0.3)]
    d = scene.cdef
    d.streching, d.shearing, d.bending, d.damping = case["stretch"], case["shear"], case["bending"], case["damping"]
    return scene, _snapshot(scene.mesh.vertices, scene.pinned, rng, case["collider"])


def _batch_scenes(case, seed):
    """Sides, stiffnesses and pins as in the batching workload, at this case's sizes."""
    scenes = b3g.batch_scenes(int(case["count"]), seed=0, side_lo=int(case["lo"]), side_hi=int(case["hi"]))
    out = []
    for k, s in enumerate(scenes):
        side = len(s.pinned)
        s.mesh = b3g.grid_mesh(side, 1.0, _jitter(side), seed * 1009 + k)
        out.append((s, _snapshot(s.mesh.vertices, s.pinned, np.random.default_rng(seed * 1013 + k), "none")))
    return out


def _requests(case, seed):
    """(scene, frames) of each request; sizes by the case, jitter and colliders by the seed."""
    sizes, rng = np.random.default_rng(11), np.random.default_rng(seed)
    out = []
    for k in range(int(case["requests"])):
        side = int(round(math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        frames = int(sizes.integers(1, int(case["most"]) + 1))
        mesh = b3g.grid_mesh(side, 1.0, _jitter(side), seed * 1019 + k)
        spheres = [((rng.uniform(-0.1, 0.1), -0.31, 0.0), 0.3, 0.3)] if k % 4 == 3 else []
        cdef = b3g.ClothDef(density=1.0, streching=1e4, shearing=1e3, damping=0.05, friction=0.3)
        pins = np.array([0, side - 1], np.uint32)
        out.append((b3g.Scene("request", mesh, cdef, pins, gravity=GRAVITY, spheres=spheres), frames))
    return out


def _block(case, seed):
    size, rng = [int(case[k]) for k in "whd"], np.random.default_rng(seed)
    scene = b3g.pinned_block_scene(*size, 1.0 / max(size))
    if not case["plastic"]:
        scene.sdef.c_yield, scene.sdef.c_creep, scene.sdef.c_max = float(np.finfo(np.float32).max), 0.0, 0.0
    p = scene.vertices.astype(np.float64)
    a, f = rng.uniform(0.004, 0.012, 3), rng.uniform(2.0, 4.0, 3)
    x = np.stack([p[:, 0] + a[0] * np.sin(f[0] * p[:, 1]), p[:, 1] + a[1] * np.sin(f[1] * p[:, 2]),
                  p[:, 2] + a[2] * np.sin(f[2] * p[:, 0])], 1)
    v = np.stack([0.2 * np.cos(f[1] * p[:, 1]), -0.5 + 0.2 * np.sin(f[2] * p[:, 0]), 0.1 * np.cos(f[0] * p[:, 2])], 1)
    v += rng.normal(0.0, 1e-3, v.shape)
    v[scene.static_nodes] = 0.0
    return scene, x.astype(np.float32), v.astype(np.float32)


def _folded(case, seed):
    """A 1 m spaced sheet of thickness 0.2 folded between two grid rows, its halves `gap` apart."""
    side, rng = int(case["side"]), np.random.default_rng(seed)
    scene = b3g.self_collision_scene(side, seed=seed % 1000003)
    x = scene.mesh.vertices.astype(np.float64)
    crease = 0.5 * (side % 2)
    half = np.where(x[:, 0] > crease, 1.0, -1.0)
    x[:, 1] = 1.6 + 0.5 * case["gap"] * half + 0.02 * np.sin(0.7 * x[:, 2]) + rng.normal(0.0, 1e-3, len(x))
    x[:, 0] = np.abs(x[:, 0] - crease)
    v = np.zeros_like(x)
    v[:, 1] = -1.0 - 0.5 * half
    v += rng.normal(0.0, 1e-2, v.shape)
    return scene, x.astype(np.float32), v.astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "cloth":
        scene, snap = _cloth_scene(case, seed)
        cloth = b3g.Cloth(scene.mesh, scene.cdef).setup(scene, _options(case["stop"], case["dot"], case["limit"]))
        if case["cg"] != "launches":
            cloth.set_cg_strategy(True, fused=case["cg"] == "fused")
        return {"case": case, "cloth": cloth, "snap": snap}
    if kind == "batch":
        built = _batch_scenes(case, seed)
        opts = _options("relative", "f64", case["limit"])
        cloths = [b3g.Cloth(s.mesh, s.cdef).setup(s, opts) for s, _ in built]
        batch = b3g.Batch(len(cloths))
        snaps = [snap for _, snap in built]
        for c, snap in zip(cloths, snaps):
            c.write_state(*snap)
        batch.autotune(cloths, DT)
        return {"case": case, "cloths": cloths, "batch": batch, "snaps": snaps}
    if kind == "server":
        server = b3g.Server(budget_bytes=2 * 10**9, max_active=256, cluster=4, split_classes=tuple(range(9, 20)))
        return {"case": case, "server": server, "requests": _requests(case, seed)}
    if kind == "softbody":
        scene, x, v = _block(case, seed)
        body = b3g.SoftBody(scene.vertices, scene.tets, scene.sdef).setup(scene)
        if case["cg"] != "persistent":
            body.set_cg_strategy(case["cg"] == "fused", fused=case["cg"] == "fused")
        q = np.zeros((len(scene.tets), 4), np.float32)
        q[:, 3] = 1.0
        return {"case": case, "body": body, "x": x, "v": v, "q": q, "eps": np.zeros((len(scene.tets), 6), np.float32)}
    scene, x, v = _folded(case, seed)
    cloth = b3g.Cloth(scene.mesh, scene.cdef).setup(scene)
    cloth.set_cg_strategy(True)
    return {"case": case, "cloth": cloth, "snap": (x, v, np.zeros_like(x))}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("cloth", "self"):
        cloth = state["cloth"]
        cloth.write_state(*state["snap"])
        for _ in range(case["frames"]):
            cloth.step(DT)
        return cloth.state()
    if kind == "batch":
        cloths, batch = state["cloths"], state["batch"]
        for c, snap in zip(cloths, state["snaps"]):
            c.write_state(*snap)
        for _ in range(case["frames"]):
            batch.step(cloths, DT)
        got = [c.state() for c in cloths]
        return {k: np.concatenate([g[k] for g in got]) for k in ("x", "v")}
    if kind == "server":
        server = state["server"]
        ids = [server.submit_scene(scene, frames) for scene, frames in state["requests"]]
        server.drain()
        got = [server.result(i) for i in ids]
        for i in ids:
            server.release(i)
        return np.concatenate(got)
    body = state["body"]
    body.write_state(state["x"], state["v"])
    body.write_elements(state["q"], state["eps"])
    for _ in range(case["frames"]):
        body.step(DT)
    return {**body.state(), **body.elements()}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------

ON_CHIP = 160e6  # bytes of L2 and shared memory: a larger system is read again in every CG iteration


def _cloth_work(n, t, springs, blocks, iterations, frames):
    """State in and out and the elements' rest data once; 40 bytes a block (values and column) in every iteration
    of a system that the chip cannot hold; about 700 operations a triangle and frame, 18 a block and iteration."""
    again = frames * iterations * 40.0 * blocks if 40.0 * blocks > ON_CHIP else 0.0
    return (77.0 * n + 40.0 * t + 24.0 * springs + again,
            frames * (700.0 * t + 80.0 * springs + iterations * (18.0 * blocks + 36.0 * n)))


def _grid_work(side, bending, iterations, frames):
    n, cells = side * side, (side - 1) ** 2
    return _cloth_work(n, 2 * cells, 3 * cells if bending else 0, (13 if bending else 7) * n, iterations, frames)


def work(case):
    kind = case["kind"]
    if kind == "cloth":
        it = case["limit"] if case["stop"] == "reference" else min(case["limit"], 30)
        parts = [_grid_work(case["side"], case["bending"], it, case["frames"])] * (2 if case["shape"] == "sewn" else 1)
    elif kind == "batch":
        sides = [len(s.pinned) for s in b3g.batch_scenes(int(case["count"]), seed=0, side_lo=int(case["lo"]),
                                                         side_hi=int(case["hi"]))]
        parts = [_grid_work(s, 0.0, min(28, case["limit"]), case["frames"]) for s in sides]
    elif kind == "server":
        parts = [_grid_work(int(math.sqrt(s.mesh.vertex_count)), 0.0, 20, f) for s, f in _requests(case, 0)]
    elif kind == "self":
        parts = [_grid_work(case["side"], 0.0, 20, case["frames"])]
    else:
        w, h, d = (int(case[k]) for k in "whd")
        n, t = (w + 1) * (h + 1) * (d + 1), 5 * w * h * d
        blocks = n + 12 * w * h * d  # the grid's edges and a diagonal on each cell face, both triangles
        # state in and out, an element's matrices (1,188 bytes) and its rotation and strain in and out
        parts = [(50.0 * n + 1268.0 * t, case["frames"] * (6000.0 * t + 20 * 18.0 * blocks))]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


# ---------------------------------------------------------------------------
# the same in 64 bits: plain torch, elements applied one by one
# ---------------------------------------------------------------------------

F64 = torch.float64


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _f64(a):
    return torch.as_tensor(np.asarray(a, np.float32).astype(np.float64), dtype=F64, device=_device())


def _f32(v):
    return float(np.float32(v))


def _outer(a, b):
    return a[..., :, None] * b[..., None, :]


def _cg(apply, diag, rhs, x0, free, stop, tol, limit, soft):
    """The filtered Jacobi-preconditioned CG; `free` is 1 on dynamic rows."""
    pinv = 1.0 / diag
    x = x0 if soft else x0 * free
    r = (rhs - apply(x)) * free
    p = z = r * pinv * free
    bh = rhs * free
    bound = float((bh * (diag if soft else pinv) * bh).sum())
    delta = float((r * z).sum())
    eps = float(np.finfo(np.float32).eps)
    mark = (eps * eps if stop == "reference" else _f32(tol) ** 2) * bound
    for _ in range(limit):
        if delta <= mark:
            break
        s = apply(p) * free
        alpha = delta / float((p * s).sum())
        x = x + alpha * p
        r = r - alpha * s
        z = r * pinv * free
        new = float((r * z).sum())
        p = z + (new / delta) * p
        delta = new
    return x


class _Sheet:
    """One cloth in 64 bits: stretch, shear and spring elements, CG, contacts with one sphere or rod."""

    def __init__(self, scene):
        mesh, d = scene.mesh, scene.cdef
        self.n = n = mesh.vertex_count
        dev = _device()
        self.tri = torch.as_tensor(mesh.triangles.astype(np.int64), device=dev)
        x = _f64(mesh.vertices)
        a, b, c = (x[self.tri[:, k]] for k in range(3))
        ab, ac = b - a, c - a
        u2 = ab.norm(dim=1)
        area2 = torch.linalg.cross(ab, ac).norm(dim=1)
        du1, dv1, du2, dv2 = u2, torch.zeros_like(u2), (ac * (ab / u2[:, None])).sum(1), area2 / u2
        inv = 1.0 / (du1 * dv2 - du2 * dv1)
        self.alpha = 0.5 * area2
        self.wu = torch.stack([inv * (dv1 - dv2), inv * dv2, -inv * dv1], 1)  # dwu/dx of the three corners
        self.wv = torch.stack([inv * (du2 - du1), -inv * du2, inv * du1], 1)
        self.mass = torch.zeros(n, dtype=F64, device=dev)
        third = (_f32(d.density) * 0.5 * area2 / 3.0)
        for k in range(3):
            self.mass.index_add_(0, self.tri[:, k], third)
        self.ks, self.kh, self.kd = _f32(d.streching), _f32(d.shearing), _f32(d.damping)
        pairs, stiff = [], []
        if d.bending > 0.0:
            pairs.append(self._bending(mesh.triangles))
            stiff.append(np.full(len(pairs[-1]), d.bending))
        if d.sewing > 0.0:
            pairs.append(mesh.sewing[:, 2:4].astype(np.int64))
            stiff.append(np.full(len(pairs[-1]), d.sewing))
        self.spring = torch.as_tensor(np.concatenate(pairs), device=dev) if pairs else None
        if pairs:
            self.spring_k = _f64(np.concatenate(stiff))
            self.spring_l = (x[self.spring[:, 0]] - x[self.spring[:, 1]]).norm(dim=1)
        self.free = torch.ones(n, 1, dtype=F64, device=dev)
        self.free[torch.as_tensor(np.asarray(scene.pinned, np.int64), device=dev)] = 0.0
        self.x, self.v, self.dv = x, torch.zeros_like(x), torch.zeros_like(x)
        self.lo, self.hi = x - EXTENSION, x + EXTENSION
        self.round = None
        if scene.spheres:
            centre, r, mu = scene.spheres[0]
            self.round = (_f64(centre), _f64(centre), _f32(r), _f32(mu))
        elif scene.capsules:
            p, q, r, mu = scene.capsules[0]
            self.round = (_f64(p), _f64(q), _f32(r), _f32(mu))
        self.exists = torch.zeros(n, dtype=torch.bool, device=dev)
        self.impulse = torch.zeros(n, 3, dtype=F64, device=dev)
        self.friction = _f32(d.friction)

    @staticmethod
    def _bending(tris):
        """The two vertices off each edge that two triangles share."""
        t = tris.astype(np.int64)
        a = np.concatenate([t[:, 0], t[:, 1], t[:, 2]])
        b = np.concatenate([t[:, 1], t[:, 2], t[:, 0]])
        c = np.concatenate([t[:, 2], t[:, 0], t[:, 1]])
        key = np.minimum(a, b) * (t.max() + 1) + np.maximum(a, b)
        order = np.argsort(key, kind="stable")
        key, c = key[order], c[order]
        same = np.nonzero(key[1:] == key[:-1])[0]
        return np.stack([c[same], c[same + 1]], 1)

    def _gather(self, p):
        return torch.stack([p[self.tri[:, k]] for k in range(3)], 1)

    def _system(self, h):
        x, v = self._gather(self.x), self._gather(self.v)
        wu = (self.wu[:, :, None] * x).sum(1)
        wv = (self.wv[:, :, None] * x).sum(1)
        alpha = self.alpha[:, None]
        force = torch.zeros_like(x)
        stiff = torch.zeros(len(x), 3, 3, 3, 3, dtype=F64, device=x.device)  # element, corner, corner, 3, 3
        damp = torch.zeros_like(stiff)
        eye = torch.eye(3, dtype=F64, device=x.device)

        def add(grad, k, c, on):
            rate = (grad * v).sum((1, 2))
            force.add_(grad * ((-k * c * on) - self.kd * rate)[:, None, None])
            blocks = grad[:, :, None, :, None] * grad[:, None, :, None, :]
            stiff.add_(blocks * (-k * on)[:, None, None, None, None])
            damp.add_(blocks, alpha=-self.kd)

        if self.kh > 0.0:
            grad = alpha[:, :, None] * (self.wu[:, :, None] * wv[:, None, :] + self.wv[:, :, None] * wu[:, None, :])
            add(grad, self.kh, self.alpha * (wu * wv).sum(1), torch.ones_like(self.alpha))
        if self.ks > 0.0:
            for w, dw in ((wu, self.wu), (wv, self.wv)):
                length = w.norm(dim=1)
                unit = w / length[:, None]
                on = (length > 1.0).to(F64)
                c = self.alpha * (length - 1.0)
                add((alpha * dw)[:, :, None] * unit[:, None, :], self.ks, c, on)
                second = (self.alpha / length * c * -self.ks * on)[:, None, None] * (eye - _outer(unit, unit))
                stiff.add_((dw[:, :, None] * dw[:, None, :])[:, :, :, None, None] * second[:, None, None])
        f = torch.zeros_like(self.x)
        for k in range(3):
            f.index_add_(0, self.tri[:, k], force[:, k])
        kv = torch.zeros_like(self.x)
        e = torch.einsum("tijab,tjb->tia", stiff, v)
        for k in range(3):
            kv.index_add_(0, self.tri[:, k], e[:, k])
        self.element = -h * damp - h * h * stiff
        del stiff, damp
        if self.spring is not None:
            p, q = self.spring[:, 0], self.spring[:, 1]
            d = self.x[p] - self.x[q]
            length = d.norm(dim=1)
            on = (length > self.spring_l).to(F64)
            dd = _outer(d, d)
            k11 = (-self.spring_k * on)[:, None, None] * (dd + (1.0 - self.spring_l / length)[:, None, None] * (eye - dd))
            rel = self.v[p] - self.v[q]
            sf = d * (-self.spring_k * on * (length - self.spring_l) / length)[:, None] - self.kd * rel
            f.index_add_(0, p, sf)
            f.index_add_(0, q, -sf)
            e = torch.einsum("sab,sb->sa", k11, rel)
            kv.index_add_(0, p, e)
            kv.index_add_(0, q, -e)
            self.link = h * self.kd * eye - h * h * k11
        f = f + self.free * self.mass[:, None] * torch.as_tensor(np.asarray(GRAVITY, np.float32).astype(np.float64),
                                                                 device=f.device)
        return h * (f + h * kv)

    def _apply(self, p):
        e = torch.einsum("tijab,tjb->tia", self.element, self._gather(p))
        out = self.mass[:, None] * p
        for k in range(3):
            out.index_add_(0, self.tri[:, k], e[:, k])
        if self.spring is not None:
            e = torch.einsum("sab,sb->sa", self.link, p[self.spring[:, 0]] - p[self.spring[:, 1]])
            out.index_add_(0, self.spring[:, 0], e)
            out.index_add_(0, self.spring[:, 1], -e)
        return out

    def _diagonal(self):
        out = self.mass[:, None].repeat(1, 3)
        for k in range(3):
            out.index_add_(0, self.tri[:, k], torch.diagonal(self.element[:, k, k], dim1=1, dim2=2))
        if self.spring is not None:
            d = torch.diagonal(self.link, dim1=1, dim2=2)
            out.index_add_(0, self.spring[:, 0], d)
            out.index_add_(0, self.spring[:, 1], d)
        return out

    def _overlaps(self):
        a, b, r, _ = self.round
        lo, hi = torch.minimum(a, b) - r - EXTENSION, torch.maximum(a, b) + r + EXTENSION
        return ((self.lo <= hi) & (self.hi >= lo)).all(1) & (self.free[:, 0] > 0)

    def step(self, stop, tol, limit):
        h = _f32(DT)
        touch = None
        if self.round is not None:
            a, b, r, mu = self.round
            self.exists &= self._overlaps()
            ab = b - a
            s = float((ab * ab).sum())
            t = ((self.x - a) @ ab / s).clamp(0.0, 1.0) if s > 0.0 else torch.zeros(self.n, dtype=F64, device=a.device)
            point = a + t[:, None] * ab
            d = self.x - point
            dist = d.norm(dim=1)
            touch = self.exists & (dist <= r)
            normal = -d / dist[:, None]  # from the particle into the shape
            big = normal[:, 0].abs() >= 0.57735027
            zero = torch.zeros_like(dist)
            t1 = torch.where(big[:, None], torch.stack([normal[:, 1], -normal[:, 0], zero], 1),
                             torch.stack([zero, normal[:, 2], -normal[:, 1]], 1))
            t2 = torch.linalg.cross(t1, normal)
        rhs = self._system(h)
        self.dv = _cg(self._apply, self._diagonal(), rhs, self.dv, self.free, stop, tol, limit, False)
        v, x = self.v + self.dv, self.x
        if touch is not None and bool(touch.any()):
            w = 1.0 / self.mass
            ni, ti, tj = (torch.where(touch, self.impulse[:, k], zero) for k in range(3))
            hit = touch[:, None]
            v = torch.where(hit, v - w[:, None] * (ni[:, None] * normal + ti[:, None] * t1 + tj[:, None] * t2), v)
            rub = math.sqrt(self.friction * mu)
            for _ in range(8):
                new = (ni + (normal * v).sum(1) / w).clamp(min=0.0)  # the particle leaves along -normal
                v = torch.where(hit, v - (w * (new - ni))[:, None] * normal, v)
                ni = torch.where(touch, new, ni)
                oi, oj = ti, tj
                ai, aj = ti + (v * t1).sum(1) / w, tj + (v * t2).sum(1) / w
                size, most = (ai * ai + aj * aj).sqrt(), rub * ni
                cut = torch.where(size > most, most / size.clamp(min=1e-300), torch.ones_like(size))
                ti, tj = torch.where(touch, ai * cut, ti), torch.where(touch, aj * cut, tj)
                v = torch.where(hit, v - w[:, None] * ((ti - oi)[:, None] * t1 + (tj - oj)[:, None] * t2), v)
            self.impulse = torch.where(hit, torch.stack([ni, ti, tj], 1), self.impulse)
        x = x + h * v
        if touch is not None and bool(touch.any()):
            for _ in range(2):
                apart = ((point - x) * normal).sum(1) - r
                push = (BAUMGARTE * (apart + SLOP)).clamp(-MAX_CORRECTION, 0.0)
                x = torch.where(touch[:, None], x + push[:, None] * normal, x)
                if float(torch.where(touch, apart, zero).min()) >= -3.0 * SLOP:
                    break
        self.x, self.v = x, v
        if self.round is not None:
            out = ~((self.lo <= x) & (x <= self.hi)).all(1, keepdim=True)
            move = 2.0 * h * v
            self.lo = torch.where(out, x - EXTENSION + move.clamp(max=0.0), self.lo)
            self.hi = torch.where(out, x + EXTENSION + move.clamp(min=0.0), self.hi)
            fresh = self._overlaps() & ~self.exists
            self.exists |= fresh
            self.impulse = torch.where(fresh[:, None], torch.zeros_like(self.impulse), self.impulse)


class _Jelly:
    """One soft body in 64 bits: corotated linear tetrahedra with plastic strain, CG of 20 iterations."""

    def __init__(self, scene):
        d, dev = scene.sdef, _device()
        self.x = _f64(scene.vertices)
        self.n = len(self.x)
        self.tet = torch.as_tensor(scene.tets.astype(np.int64), device=dev)
        p = self.x[self.tet]
        self.rest = p
        edges = torch.stack([p[:, k] - p[:, 0] for k in (1, 2, 3)], 2)  # columns
        volume = torch.linalg.det(edges).abs() / 6.0
        self.inv = torch.linalg.inv(edges)
        mass = _f32(d.density) * volume
        self.mass = torch.zeros(self.n, dtype=F64, device=dev)
        for k in range(4):
            self.mass.index_add_(0, self.tet[:, k], 0.25 * mass)
        e, nu = _f32(d.E), _f32(d.nu)
        lam, mu = nu * e / ((1 + nu) * (1 - 2 * nu)), e / (2 * (1 + nu))
        mat = torch.zeros(6, 6, dtype=F64, device=dev)
        mat[:3, :3] = lam
        for k in range(3):
            mat[k, k] = lam + 2 * mu
            mat[3 + k, 3 + k] = mu
        grad = torch.cat([self.inv.sum(1, keepdim=True), -self.inv], 1)  # strains count compression positive
        self.strain = torch.zeros(len(p), 6, 4, 3, dtype=F64, device=dev)
        for r, (i, j) in enumerate([(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]):
            self.strain[:, r, :, i] = grad[:, :, j]
            if i != j:
                self.strain[:, r, :, j] = grad[:, :, i]
        flat = self.strain.reshape(-1, 6, 12)
        stress = volume[:, None, None] * (flat.transpose(1, 2) @ mat)
        self.ke = (stress @ flat).reshape(-1, 4, 3, 4, 3)
        self.plastic_force = stress.reshape(-1, 4, 3, 6)
        self.free = torch.ones(self.n, 1, dtype=F64, device=dev)
        self.free[torch.as_tensor(np.asarray(scene.static_nodes, np.int64), device=dev)] = 0.0
        self.damping = _f64(scene.mass_damping)
        self.limits = _f32(d.c_yield), _f32(d.c_creep), _f32(d.c_max)
        self.eps = torch.zeros(len(p), 6, dtype=F64, device=dev)
        self.q = torch.zeros(len(p), 4, dtype=F64, device=dev)
        self.q[:, 3] = 1.0

    @staticmethod
    def _matrix(q):
        x, y, z, w = q.unbind(1)
        return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                            2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                            2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)

    def step(self):
        h, tet = _f32(DT), self.tet
        p = self.x[tet]
        a = torch.stack([p[:, k] - p[:, 0] for k in (1, 2, 3)], 2) @ self.inv
        q = self.q
        for _ in range(20):
            r = self._matrix(q)
            s = (r * a).sum((1, 2)).abs()
            omega = torch.linalg.cross(r, a, dim=1).sum(2) * (1.0 / s + 1e-9)[:, None]
            w = omega.norm(dim=1, keepdim=True)
            axis = omega / w.clamp(min=1e-300)
            half = torch.cat([torch.sin(0.5 * w) * axis, torch.cos(0.5 * w)], 1)
            (x1, y1, z1, w1), (x2, y2, z2, w2) = half.unbind(1), q.unbind(1)
            new = torch.stack([w1 * x2 + x1 * w2 + y1 * z2 - z1 * y2, w1 * y2 + y1 * w2 + z1 * x2 - x1 * z2,
                               w1 * z2 + z1 * w2 + x1 * y2 - y1 * x2, w1 * w2 - x1 * x2 - y1 * y2 - z1 * z2], 1)
            q = torch.where(w < 1e-9, q, new / new.norm(dim=1, keepdim=True))
        self.q = q
        r = self._matrix(q)
        back = torch.einsum("eba,ekb->eka", r, p) - self.rest
        yields, creep, most = self.limits
        elastic = torch.einsum("erkc,ekc->er", self.strain, back) - self.eps
        flows = (elastic.norm(dim=1, keepdim=True) > yields).to(F64)
        eps = self.eps + flows * h * min(creep, 1.0 / h) * elastic
        size = eps.norm(dim=1, keepdim=True)
        self.eps = torch.where(size > most, eps * (most / size.clamp(min=1e-300)), eps)
        flow = torch.einsum("eab,ekbr,er->eka", r, self.plastic_force, self.eps)
        block = torch.einsum("eab,eibjc,edc->eiajd", r, self.ke, r)
        f0 = torch.einsum("eab,eibjc,ejc->eia", r, self.ke, self.rest)

        def spread(e):
            out = torch.zeros(self.n, 3, dtype=F64, device=e.device)
            for k in range(4):
                out.index_add_(0, tet[:, k], e[:, k])
            return out

        g = torch.as_tensor(np.asarray(GRAVITY, np.float32).astype(np.float64), device=self.x.device)
        m = self.mass[:, None]
        stretch = spread(torch.einsum("eiajd,ejd->eia", block, p))
        rhs = m * self.v - h * (stretch - spread(f0) - spread(flow) - self.free * m * g)
        scale = m + h * self.damping[:, None] * m

        def apply(y):
            return scale * y + h * h * spread(torch.einsum("eiajd,ejd->eia", block, y[tet]))

        diag = scale + h * h * spread(torch.diagonal(torch.stack([block[:, k, :, k] for k in range(4)], 1), dim1=2,
                                                     dim2=3))
        self.v = _cg(apply, diag, rhs, self.v, self.free, "reference", 0.0, 20, True)
        self.x = self.x + h * self.v


def _numpy(t):
    return t.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "self":
        return None  # thousands of contacts solved one after another in list order: minutes in plain Python
    if kind == "cloth":
        scene, snap = _cloth_scene(case, seed)
        sheet = _Sheet(scene)
        sheet.x, sheet.v, sheet.dv = (_f64(a) for a in snap)
        for _ in range(case["frames"]):
            sheet.step(case["stop"], 1e-4, case["limit"])
        return {"x": _numpy(sheet.x), "v": _numpy(sheet.v), "dv": _numpy(sheet.dv)}
    if kind == "batch":
        sheets = []
        for scene, snap in _batch_scenes(case, seed):
            sheet = _Sheet(scene)
            sheet.x, sheet.v, sheet.dv = (_f64(a) for a in snap)
            for _ in range(case["frames"]):
                sheet.step("relative", 1e-4, case["limit"])
            sheets.append(sheet)
        return {k: np.concatenate([_numpy(getattr(s, k)) for s in sheets]) for k in ("x", "v")}
    if kind == "server":
        out = []
        for scene, frames in _requests(case, seed):
            sheet = _Sheet(scene)
            for _ in range(frames):
                sheet.step("relative", 1e-4, 200)
            out.append(_numpy(sheet.x))
        return np.concatenate(out)
    scene, x, v = _block(case, seed)
    jelly = _Jelly(scene)
    jelly.x, jelly.v = _f64(x), _f64(v)
    for _ in range(case["frames"]):
        jelly.step()
    return {k: _numpy(getattr(jelly, k)) for k in ("x", "v", "q", "eps")}
