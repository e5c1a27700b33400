"""The cooperative CG kernels (grid_cg.cu) on the systems that the on-chip CG
leaves to them -- a vertex of many neighbours, and large cloths in random
numbering (resident_shape_check.cpp checks that it does) -- against 64-bit solves
and the oracle on the CPU."""
import ctypes as C

import numpy as np
import pytest

from helpers import rel_err
from numberings import hub_body_scene, hub_mesh, renumbered, rounding_bound, scene_of, solve64

pytestmark = pytest.mark.gpu

ITERATIONS = 8


def _scene(b3g, kind, size, bending):
    if kind == "hub":
        return scene_of(b3g, hub_mesh(b3g, 20 if bending else 40, size), bending)
    return scene_of(b3g, renumbered(b3g.grid_mesh(size, 1.0, 1e-3, 1), np.random.default_rng(size)), bending)


# rows of 41 blocks; one row a thread with its blocks in shared memory (240^2) and
# without (268^2, 13 blocks a row); several rows a thread
@pytest.mark.parametrize("kind,size,bending", [("hub", 30, 0.0), ("hub", 30, 1e2), ("random", 240, 0.0),
                                               ("random", 268, 1e2), ("random", 300, 0.0)])
@pytest.mark.parametrize("dot", [0, 2])
def test_cooperative_cg_matches_64_bits(b3g, port, kind, size, bending, dot):
    """The one-pass form rounds beta's numerator apart from the oracle: to the
    bound of the two-pass form comes one more rounding an iteration (1e-5 of
    the largest entry, as for the streamed matrices)."""
    scene = _scene(b3g, kind, size, bending)
    v = np.random.default_rng(size).normal(0.0, 0.1, (scene.mesh.vertex_count, 3)).astype(np.float32)
    v[0] = 0.0
    exact = None
    for persistent, fused in ((False, False), (True, False), (True, True)):
        cloth = b3g.Cloth(scene.mesh, scene.cdef).setup(scene, b3g.SolverOptions(b3g.STOP_RELATIVE, 1e-9, ITERATIONS, dot))
        cloth.set_cg_strategy(persistent, fused)
        cloth.write_state(v=v, dv=0.1 * v)
        if exact is None:
            cloth.assemble(scene.dt)
            system = cloth.system()
            exact = solve64(system, ITERATIONS)
            bound = rounding_bound(port, system, ITERATIONS, dot, exact)
        assert cloth.step(scene.dt)["iterations"] == ITERATIONS
        far = np.abs(cloth.state()["dv"] - exact).max()
        assert far <= bound + (1e-5 * np.abs(exact).max() if fused else 0.0), (persistent, fused)


@pytest.mark.parametrize("form", ["persistent", "fused"])
@pytest.mark.parametrize("dot", [0, 2])
def test_cooperative_cg_of_a_softbody(b3g, port, dot, form):
    """The soft body mode of both forms, a step at a time from identical state
    (the tolerances of test_softbody_step_matches_oracle)."""
    scene = hub_body_scene(b3g)
    s = scene.sdef
    opts = b3g.SolverOptions.reference() if dot == 0 else b3g.SolverOptions.relative(1e-5, 200, dot)
    gpu = b3g.SoftBody(scene.vertices, scene.tets, s).setup(scene, opts)
    gpu.set_cg_strategy(True, fused=form == "fused")
    ora = port.PortSoftBody(scene.vertices, scene.tets, s.density, s.E, s.nu, s.c_yield, s.c_creep, s.c_max).setup(scene)
    ora.set_solver(opts.stop_rule, opts.tolerance, opts.max_iterations, opts.dot)
    for step in range(20):
        st, el = gpu.state(), gpu.elements()
        ora.set_state(x=st["x"], v=st["v"])
        ora.set_elements(q=el["q"], eps=el["eps"])
        if step % 9 == 0:
            gpu.apply_force(11, [0.0, 60.0, 5.0])
            ora.apply_force(11, [0.0, 60.0, 5.0])
        g = gpu.step(scene.dt)
        o = ora.step(scene.dt)
        assert abs(g["iterations"] - o["iterations"]) <= 1, (step, g["iterations"], o["iterations"])
        assert rel_err(gpu.state()["x"], ora.state()["x"]) <= 1e-4, step
        assert rel_err(gpu.state()["v"], ora.state()["v"]) <= 1e-4, step


@pytest.mark.parametrize("fused", [False, True])
def test_cooperative_cg_bounded_wait_times_out(b3g, fused):
    """The counter barrier that never completes ends in B3G_ERR_TIMEOUT, and the
    next step is that of a cloth that never met one."""
    scene = _scene(b3g, "hub", 100, 0.0)
    ends = []
    for waits in (True, False):
        cloth = b3g.Cloth(scene.mesh, scene.cdef).setup(scene, b3g.SolverOptions.relative(1e-4, 50))
        cloth.set_cg_strategy(True, fused=fused)
        if waits:
            res = C.c_int(0)
            b3g.check(b3g.lib().b3g_debug_cg_barrier_timeout(cloth.h, 2000, C.byref(res)), "timeout diag")
            assert res.value == 7  # B3G_ERR_TIMEOUT
        assert cloth.step(scene.dt)["iterations"] > 0
        ends.append(cloth.state()["dv"])
    assert np.array_equal(ends[0], ends[1])
