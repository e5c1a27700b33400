"""State transfers: what is written is read back bit for bit, on both sides of
the largest staged call, for odd vertex counts, partial calls and float patterns
that arithmetic would not keep (NaN payloads, negative zero, denormals)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _words(rng, shape):
    return rng.integers(0, 2**32, shape, dtype=np.uint32).view(np.float32)


# tiles of 256 vertices: below, at and past one; the last staged write (147^2) and
# read (835^2) and the first that are not
@pytest.mark.parametrize("side", [2, 15, 16, 17, 147, 148, 835, 836])
def test_cloth_state_round_trip(b3g, side):
    cloth = b3g.Cloth(b3g.grid_mesh(side, 1.0), b3g.ClothDef(density=1.0))
    rng = np.random.default_rng(side)
    x, v, dv = (_words(rng, (cloth.n, 3)) for _ in range(3))
    cloth.write_state(x, v, dv)
    for got, want in zip(cloth.state().values(), (x, v, dv)):
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    cloth.write_state(v=x)  # one array alone: the others keep theirs
    for got, want in zip(cloth.state().values(), (x, x, dv)):
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert np.array_equal(cloth.positions().view(np.uint32), x.view(np.uint32))


@pytest.mark.parametrize("side", [1, 7, 16, 18])
def test_softbody_state_round_trip(b3g, side):
    scene = b3g.pinned_block_scene(side, side, side, 1.0 / side)
    body = b3g.SoftBody(scene.vertices, scene.tets, scene.sdef)
    rng = np.random.default_rng(side)
    x, v = _words(rng, scene.vertices.shape), _words(rng, scene.vertices.shape)
    q, eps = _words(rng, (len(scene.tets), 4)), _words(rng, (len(scene.tets), 6))
    body.write_state(x, v)
    body.write_elements(q, eps)
    for got, want in zip([*body.state().values(), *body.elements().values()], (x, v, q, eps)):
        assert np.array_equal(got.view(np.uint32).ravel(), want.view(np.uint32).ravel())
