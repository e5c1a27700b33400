"""Cloths whose vertices are not numbered row by row, and the filtered CG in 64
bits on the CPU: an answer that none of the GPU's CG forms had a part in."""
import dataclasses

import numpy as np


def renumbered(mesh, rng):
    """The mesh with its vertices in random order."""
    order = rng.permutation(mesh.vertex_count)
    new = np.empty_like(order)
    new[order] = np.arange(order.size)
    return dataclasses.replace(mesh, vertices=mesh.vertices[order], triangles=new[mesh.triangles].astype(np.uint32))


def tube_mesh(b3g, rows, side):
    """rows x side vertices, the last row joined to the first one."""
    angle = 2.0 * np.pi * np.arange(rows) / rows
    vertices = np.zeros((rows, side, 3))
    vertices[:, :, 0] = np.linspace(-0.5, 0.5, side)
    vertices[:, :, 1] = np.sin(angle)[:, None] / (2.0 * np.pi)
    vertices[:, :, 2] = np.cos(angle)[:, None] / (2.0 * np.pi)
    i, j = (k.ravel() for k in np.meshgrid(np.arange(rows), np.arange(side - 1), indexing="ij"))
    a, b = i * side + j, (i + 1) % rows * side + j
    tris = np.concatenate([np.stack([b + 1, b, a], 1), np.stack([a, a + 1, b + 1], 1)])
    return b3g.Mesh(vertices.reshape(-1, 3).astype(np.float32), tris.astype(np.uint32))


def hub_mesh(b3g, spokes, rings):
    """A disc: one vertex coupled to `spokes` others, in `rings` rings."""
    angle = 2.0 * np.pi * np.arange(spokes) / spokes
    radius = 0.5 * np.arange(1, rings + 1) / rings
    ring = radius[:, None, None] * np.stack([np.cos(angle), np.zeros(spokes), np.sin(angle)], 1)[None]
    k, s = (q.ravel() for q in np.meshgrid(np.arange(rings - 1), np.arange(spokes), indexing="ij"))
    t = (s + 1) % spokes
    a, b, c, d = 1 + k * spokes + s, 1 + k * spokes + t, 1 + (k + 1) * spokes + s, 1 + (k + 1) * spokes + t
    hub = np.stack([np.zeros(spokes), 1 + (np.arange(spokes) + 1) % spokes, 1 + np.arange(spokes)], 1)
    tris = np.concatenate([hub, np.stack([a, b, d], 1), np.stack([a, d, c], 1)])
    return b3g.Mesh(np.concatenate([np.zeros((1, 3)), ring.reshape(-1, 3)]).astype(np.float32), tris.astype(np.uint32))


def scene_of(b3g, mesh, bending=0.0, pinned=(0,)):
    cdef = b3g.ClothDef(density=1.0, streching=1e4, shearing=1e3, bending=bending, damping=0.05, friction=0.3)
    return b3g.Scene("mesh", mesh, cdef, np.asarray(pinned, np.uint32))


def solve64(system, iterations):
    """x after so many iterations of b3SolveMPCG (src/bounce/cloth/
    cloth_force_solver.cpp:61-136) on an exported system, in 64 bits."""
    import scipy.sparse

    n = system["rowptr"].size - 1
    vals = system["vals"].astype(np.float64).reshape(-1, 3, 3).transpose(0, 2, 1)  # stored by columns
    A = scipy.sparse.bsr_array((vals, system["cols"].astype(np.int64), system["rowptr"].astype(np.int64)),
                               shape=(3 * n, 3 * n)).tocsr()
    S = np.repeat(system["S"].astype(np.float64), 3)
    P = 1.0 / A.diagonal()
    x = S * system["x0"].astype(np.float64)
    r = S * (system["b"].astype(np.float64) - A @ x)
    p = z = S * P * r
    delta = r @ z
    for _ in range(iterations):
        s = S * (A @ p)
        alpha = delta / (p @ s)
        x = x + alpha * p
        r = r - alpha * s
        z = S * P * r
        new = r @ z
        p = z + new / delta * p
        delta = new
    return x.reshape(-1, 3)


def rounding_bound(port, system, iterations, dot, exact):
    """How far a solve in 32 bits may be from the 64-bit one: four times as far
    as the oracle's (the same algorithm, its sums in another order, its roundings
    as many and as large), and at least 1e-6 of the largest entry."""
    x, it, _ = port.mpcg(system, 1, 1e-9, iterations, dot)
    assert it == iterations
    return max(4.0 * np.abs(x - exact).max(), 1e-6 * np.abs(exact).max())


def hub_body_scene(b3g):
    """A ball of tetrahedra around one node: an icosahedron's faces split in
    four, 42 nodes on the surface, each of them coupled to the centre."""
    g = (1.0 + np.sqrt(5.0)) / 2.0
    points = [np.array(p) for a in (-1.0, 1.0) for b in (-g, g) for p in ((0, a, b), (a, b, 0), (b, 0, a))]
    faces = []
    for i in range(12):
        for j in range(i + 1, 12):
            for k in range(j + 1, 12):
                if max(np.linalg.norm(points[i] - points[j]), np.linalg.norm(points[j] - points[k]),
                       np.linalg.norm(points[k] - points[i])) < 2.1:
                    faces.append((i, j, k))
    middle = {}
    for f in faces:
        for a, b in ((f[0], f[1]), (f[1], f[2]), (f[0], f[2])):
            if (a, b) not in middle:
                middle[(a, b)] = len(points)
                points.append(0.5 * (points[a] + points[b]))
    tets = []
    vertices = np.array([np.zeros(3)] + [p / np.linalg.norm(p) for p in points])
    for i, j, k in faces:
        a, b, c = middle[(i, j)], middle[(j, k)], middle[(i, k)]
        for t in ((i, a, c), (a, j, b), (c, b, k), (a, b, c)):
            p, q, r = (vertices[1 + m] for m in t)
            t = t if np.dot(p, np.cross(q, r)) > 0.0 else (t[0], t[2], t[1])
            tets.append((0, 1 + t[0], 1 + t[1], 1 + t[2]))
    sdef = b3g.SoftBodyDef(density=0.2, E=1000.0, nu=0.33, c_yield=0.1, c_creep=0.5, c_max=1.0)
    pin = int(np.argmax(vertices[:, 1]))
    return b3g.SoftBodyScene(vertices.astype(np.float32), np.asarray(tets, np.uint32), sdef,
                             np.full(len(vertices), 0.2, np.float32), np.array([pin], np.uint32))
