"""The on-chip CG of one cloth against the per-iteration kernels: the same
rows, so with FP64 dots the same floats but for the sums' last bits.

Sizes sit on the edges of its shapes: one CTA (up to 256 rows), clusters (a
last CTA with few rows or none, 4,096 rows), the grid (one and two rows a
thread, blocks that do not all fit), and a coupling across the whole cloth
(sewn panels)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(b3g, kind, side):
    if kind == "sewn":
        return b3g.sewn_scene(side)
    if kind == "bend":
        return b3g.sphere_scene(side)
    return b3g.plain_scene(side)


@pytest.mark.parametrize("kind,side", [("plain", 2), ("plain", 6), ("bend", 16), ("plain", 17), ("bend", 33),
                                       ("plain", 64), ("plain", 65), ("sewn", 9), ("sewn", 45), ("sewn", 50),
                                       ("bend", 67), ("bend", 250), ("plain", 280), ("plain", 384)])
@pytest.mark.parametrize("dot", [0, 1, 2])
def test_on_chip_cg_matches_launches(b3g, kind, side, dot):
    """x of an iteration differs only by the rounding of alpha and beta, one
    float rounding (6e-8) each and iteration, magnified by at most the CG's own
    sensitivity; 8 iterations of both from the same system stay within 1e-5 of
    the largest entry (FP64 sums: within 1e-6)."""
    scene = _scene(b3g, kind, side)
    opts = b3g.SolverOptions(b3g.STOP_RELATIVE, 1e-9, 3 if side == 2 else 8, dot)
    rng = np.random.default_rng(side)
    v = rng.normal(0.0, 0.1, (scene.mesh.vertex_count, 3)).astype(np.float32)
    v[np.asarray(scene.pinned, np.int64)] = 0.0
    got = []
    for persistent in (False, True):
        cloth = b3g.Cloth(scene.mesh, scene.cdef).setup(scene, opts)
        cloth.set_cg_strategy(persistent)
        cloth.write_state(v=v, dv=0.1 * v)
        out = cloth.step_profiled(scene.dt)
        got.append((out["iterations"], cloth.state()["dv"]))
        again = cloth.step(scene.dt)
        assert again["iterations"] > 0
    assert got[0][0] == got[1][0]
    a, b = got[0][1].astype(np.float64), got[1][1].astype(np.float64)
    assert np.abs(a - b).max() <= (1e-6 if dot == 2 else 1e-5) * np.abs(a).max()


@pytest.mark.parametrize("kind,side", [("plain", 517), ("plain", 577), ("bend", 450)])
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("dot", [0, 2])
def test_streamed_matrix_matches_launches(b3g, kind, side, fused, dot):
    """Cloths whose matrix does not stay in L2 (a last slice that is not full;
    rows with and without bending), with the same bound; the one-pass form
    rounds beta's numerator apart, one more rounding an iteration."""
    scene = _scene(b3g, kind, side)
    opts = b3g.SolverOptions(b3g.STOP_RELATIVE, 1e-9, 8, dot)
    rng = np.random.default_rng(side)
    v = rng.normal(0.0, 0.1, (scene.mesh.vertex_count, 3)).astype(np.float32)
    v[np.asarray(scene.pinned, np.int64)] = 0.0
    got = []
    for persistent in (False, True):
        cloth = b3g.Cloth(scene.mesh, scene.cdef).setup(scene, opts)
        cloth.set_cg_strategy(persistent, fused and persistent)
        cloth.write_state(v=v, dv=0.1 * v)
        cloth.step(scene.dt)
        got.append(cloth.state()["dv"].astype(np.float64))
        cloth.close()
    assert np.abs(got[0] - got[1]).max() <= 1e-5 * np.abs(got[0]).max()


def test_on_chip_cg_repeats_itself(b3g):
    """The grid form's sums run in a fixed order: the same step twice gives the
    same bits."""
    scene = b3g.plain_scene(128)
    cloth = b3g.Cloth(scene.mesh, scene.cdef).setup(scene, b3g.SolverOptions.relative(1e-4, 50, b3g.DOT_F32))
    cloth.set_cg_strategy(True)
    x0 = cloth.state()
    runs = []
    for _ in range(3):
        cloth.write_state(x0["x"], x0["v"], x0["dv"])
        cloth.step(scene.dt)
        cloth.step(scene.dt)
        runs.append(cloth.state()["dv"])
    assert all(np.array_equal(runs[0], r) for r in runs[1:])


@pytest.mark.parametrize("cluster,split", [(1, ()), (8, tuple(range(32)))])
@pytest.mark.parametrize("dot", [0, 2])
def test_batch_on_chip_matches_launches(b3g, cluster, split, dot):
    """Cloths at the edges of the batch's on-chip forms (one, two and four rows
    a thread on one CTA and on a cluster, bending rows, a sewn pair, and one
    past its reach): the same bound as above against each cloth stepped alone
    with the per-iteration kernels or the on-chip CG."""
    opts = b3g.SolverOptions(b3g.STOP_RELATIVE, 1e-9, 8, dot)
    scenes = [b3g.plain_scene(2 if k == 0 else s) for k, s in enumerate((2, 22, 23, 32, 33, 45, 46, 64, 65, 91))]
    scenes += [b3g.sphere_scene(22), b3g.sphere_scene(40), b3g.sewn_scene(20), b3g.plain_scene(130)]
    small = b3g.SolverOptions(b3g.STOP_RELATIVE, 1e-9, 3, dot)
    alone, cloths = [], []
    for k, scene in enumerate(scenes):
        rng = np.random.default_rng(k)
        v = rng.normal(0.0, 0.1, (scene.mesh.vertex_count, 3)).astype(np.float32)
        v[np.asarray(scene.pinned, np.int64)] = 0.0
        for where in (alone, cloths):
            c = b3g.Cloth(scene.mesh, scene.cdef).setup(scene, small if k == 0 else opts)
            c.write_state(v=v, dv=0.1 * v)
            where.append(c)
    batch = b3g.Batch(len(cloths))
    batch.set_schedule(cluster, split)
    batch.step(cloths, scenes[0].dt)
    for a, b in zip(alone, cloths):
        a.step(scenes[0].dt)
        x, y = a.state()["dv"].astype(np.float64), b.state()["dv"].astype(np.float64)
        assert np.abs(x - y).max() <= (1e-6 if dot == 2 else 1e-5) * np.abs(x).max()


@pytest.mark.parametrize("side", [91, 280])
def test_withheld_rows_time_out(b3g, side):
    """The grid form's waits for partials and, in the diagnostic's second run, for
    rows of z alone end in B3G_ERR_TIMEOUT, and the next step is that of a cloth
    that never met one."""
    import ctypes as C

    scene = b3g.plain_scene(side)
    ends = []
    for waits in (True, False):
        cloth = b3g.Cloth(scene.mesh, scene.cdef).setup(scene, b3g.SolverOptions.relative(1e-4, 50))
        cloth.set_cg_strategy(True)
        if waits:
            res = C.c_int(0)
            b3g.check(b3g.lib().b3g_debug_cg_barrier_timeout(cloth.h, 2000, C.byref(res)), "timeout diag")
            assert res.value == 7  # B3G_ERR_TIMEOUT
        assert cloth.step(scene.dt)["iterations"] > 0
        ends.append(cloth.state()["dv"])
    assert np.array_equal(ends[0], ends[1])
