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
