"""Launches shorter than the GPU, over every tree layout and both triangle
tests: the oracle's answers bit for bit."""
import numpy as np
import pytest

from ajisai_render_gb300 import api
from ajisai_render_gb300 import scenes as S
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def flat():
    return S.flatten(S.icosphere_scene(subdiv=4, seed=3, width=8, height=8))


@pytest.mark.parametrize("tri_test", [0, 1])
@pytest.mark.parametrize("width", [2, 4, 8, 0x104, 0x108])
def test_short_queues_match_the_oracle(ctx, flat, tri_test, width):
    scene = api.GpuScene(ctx, flat, api.CreatePLOCAggregate(14, tri_test, bvh_width=width))
    rng = np.random.default_rng(7)
    m = 5473
    o = rng.uniform(-2, 2, (m, 3))
    d = rng.uniform(-1, 1, (m, 3)) - o
    far = np.where(rng.uniform(size=(m, 1)) < 0.3, 0.9, np.inf)
    rays = np.concatenate([o, d, np.full((m, 1), 1e-4), far], 1).astype(np.float32)
    ot, op, ou, ov = O.trace(flat.tris, rays, tri_test=tri_test)  # every triangle
    occ = O.trace(flat.tris, rays, any_hit=True, tri_test=tri_test)[1] == 1
    assert 0.1 < (op >= 0).mean() < 0.95
    # one ray, around a warp, around one ray a warp of the resident blocks
    for n in (1, 31, 33, 4865, 5473):
        t, p, u, v = scene.Intersect(rays[:n])
        assert np.array_equal(p, op[:n])
        hit = p >= 0
        for got, want in ((t, ot), (u, ou), (v, ov)):
            assert np.array_equal(got[hit].view(np.uint32), want[:n][hit].view(np.uint32))
        assert np.array_equal(scene.Occlude(rays[:n]), occ[:n])
