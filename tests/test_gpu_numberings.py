"""The on-chip CG against a 64-bit solve on the CPU, on grids and on
cloths whose couplings reach across the whole numbering -- closed tubes and
grids in random order.  A CTA (resident_cg.cuh) keeps the whole band of its rows:
a last CTA of few rows has the most rows outside its own."""
import numpy as np
import pytest

from numberings import renumbered, rounding_bound, scene_of, solve64, tube_mesh

pytestmark = pytest.mark.gpu

ITERATIONS = 8


def _mesh(b3g, kind, rows, side):
    if kind == "tube":
        return tube_mesh(b3g, rows, side)
    return renumbered(b3g.grid_mesh(side, 1.0, 1e-3, 1), np.random.default_rng(side))


def _cloth(b3g, scene, dot, seed, iterations=ITERATIONS):
    """A cloth in motion, as every call with the same arguments makes it."""
    cloth = b3g.Cloth(scene.mesh, scene.cdef).setup(scene, b3g.SolverOptions(b3g.STOP_RELATIVE, 1e-9, iterations, dot))
    v = np.random.default_rng(seed).normal(0.0, 0.1, (cloth.n, 3)).astype(np.float32)
    v[np.asarray(scene.pinned, np.int64)] = 0.0
    cloth.write_state(v=v, dv=0.1 * v)
    return cloth


def _exact(port, cloth, scene, dot, iterations=ITERATIONS):
    """The 64-bit solve of the system that the cloth's next step solves, and its bound."""
    cloth.assemble(scene.dt)
    system = cloth.system()
    exact = solve64(system, iterations)
    return exact, rounding_bound(port, system, iterations, dot, exact)


# One CTA, clusters (a last CTA with few rows or none, 4,096 rows), the grid, rows
# with bending, and sewn panels: a cloth of up to 4,096 vertices runs the same
# on-chip kernel under every strategy, so only another solve can tell.
@pytest.mark.parametrize("maker,side", [("plain", 2), ("plain", 6), ("sphere", 16), ("plain", 17), ("sphere", 33),
                                        ("plain", 64), ("plain", 65), ("sewn", 9), ("sewn", 45), ("sewn", 50),
                                        ("sphere", 67), ("plain", 280)])
@pytest.mark.parametrize("dot", [0, 1, 2])
def test_on_chip_cg_matches_64_bits(b3g, port, maker, side, dot):
    scene = getattr(b3g, f"{maker}_scene")(side)
    iterations = 3 if side == 2 else ITERATIONS
    exact = bound = None
    for persistent in (False, True):
        cloth = _cloth(b3g, scene, dot, side, iterations)
        cloth.set_cg_strategy(persistent)
        if exact is None:
            exact, bound = _exact(port, cloth, scene, dot, iterations)
        assert cloth.step(scene.dt)["iterations"] == iterations
        assert np.abs(cloth.state()["dv"] - exact).max() <= bound


@pytest.mark.parametrize("kind,rows,side", [("tube", 27, 27), ("tube", 33, 32), ("tube", 46, 46), ("tube", 48, 48),
                                            ("tube", 64, 64), ("random", 34, 34), ("random", 40, 40),
                                            ("random", 46, 46), ("random", 64, 64), ("tube", 91, 91),
                                            ("random", 91, 91)])
@pytest.mark.parametrize("dot", [0, 2])
def test_wide_numberings_match_64_bits(b3g, port, kind, rows, side, dot):
    scene = scene_of(b3g, _mesh(b3g, kind, rows, side))
    exact = bound = None
    for persistent, fused in ((False, False), (True, False), (True, True)):
        cloth = _cloth(b3g, scene, dot, side)
        cloth.set_cg_strategy(persistent, fused)
        if exact is None:
            exact, bound = _exact(port, cloth, scene, dot)
        assert cloth.step(scene.dt)["iterations"] == ITERATIONS
        assert np.abs(cloth.state()["dv"] - exact).max() <= bound


# 48 x 48: the band in reach of eight CTAs but for the last one's; 52 x 52: of four
@pytest.mark.parametrize("cluster", [1, 4, 8])
@pytest.mark.parametrize("dot", [0, 2])
def test_wide_numberings_in_a_batch(b3g, port, cluster, dot):
    scenes = [scene_of(b3g, _mesh(b3g, kind, side, side))
              for kind, side in (("tube", 27), ("tube", 46), ("tube", 48), ("tube", 52), ("random", 34), ("random", 48))]
    cloths = [_cloth(b3g, s, dot, k) for k, s in enumerate(scenes)]
    want = [_exact(port, c, s, dot) for c, s in zip(cloths, scenes)]
    batch = b3g.Batch(len(cloths))
    batch.set_schedule(cluster, tuple(range(32)) if cluster > 1 else ())
    batch.step(cloths, scenes[0].dt)
    for cloth, (exact, bound) in zip(cloths, want):
        assert np.abs(cloth.state()["dv"] - exact).max() <= bound
