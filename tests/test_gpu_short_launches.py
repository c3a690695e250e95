"""Launches shorter than the GPU: a traversal spreads a short queue over all
its warps, and its answers are those of the same rays in a long queue."""
import numpy as np
import pytest

from ajisai_render_gb300 import api
from ajisai_render_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    ctx = api.Context(0)
    flat = S.flatten(S.icosphere_scene(subdiv=5, seed=3, width=8, height=8))
    yield api.GpuScene(ctx, flat)
    ctx.close()


# one ray, around a warp, around one ray a warp (8 or 9 blocks of 4 warps on
# 152 SMs) and around one ray a lane
@pytest.mark.parametrize("n", [1, 31, 33, 4863, 4865, 5471, 5473, 155_647, 155_649, 175_105])
def test_short_queues_give_the_long_queues_answers(scene, n):
    rng = np.random.default_rng(2)
    m = 200_000
    o = rng.uniform(-2, 2, (m, 3))
    d = rng.uniform(-1, 1, (m, 3)) - o
    far = np.where(rng.uniform(size=(m, 1)) < 0.3, 0.9, np.inf)
    rays = np.concatenate([o, d, np.full((m, 1), 1e-4), far], 1).astype(np.float32)
    for a, b in zip(scene.Intersect(rays[:n]), scene.Intersect(rays)):
        assert np.array_equal(a, b[:n])
    assert np.array_equal(scene.Occlude(rays[:n]), scene.Occlude(rays)[:n])
