"""Host ray queries large enough to run in parts (from 2 x 786,432 rays on,
in two to four): the answers of the same rays in whole calls, bit for bit, also
behind a render that is still running on the context."""
import numpy as np
import pytest

from ajisai_render_gb300 import api
from ajisai_render_gb300 import scenes as S

pytestmark = pytest.mark.gpu

PART = 3 << 18
MOST = 4 * PART + 5


@pytest.fixture(scope="module")
def made():
    """The scene, the rays, and their answers in calls of less than two parts."""
    ctx = api.Context(0)
    flat = S.flatten(S.icosphere_scene(subdiv=4, seed=5, width=512, height=512))
    scene = api.GpuScene(ctx, flat)
    rng = np.random.default_rng(11)
    o = rng.uniform(-2, 2, (MOST, 3)).astype(np.float32)
    d = rng.uniform(-1, 1, (MOST, 3)).astype(np.float32) - o
    far = np.where(rng.uniform(size=(MOST, 1)) < 0.3, 0.9, np.inf)
    rays = np.concatenate([o, d, np.full((MOST, 1), 1e-4), far], 1).astype(np.float32)
    step = 1_000_003
    hits = [scene.Intersect(rays[k:k + step]) for k in range(0, MOST, step)]
    closest = [np.concatenate(x) for x in zip(*hits)]
    occluded = np.concatenate([scene.Occlude(rays[k:k + step]) for k in range(0, MOST, step)])
    yield ctx, scene, rays, closest, occluded
    ctx.close()


def check(made, n):
    _, scene, rays, closest, occluded = made
    for got, want in zip(scene.Intersect(rays[:n]), closest):
        assert np.array_equal(got.view(np.uint32), want[:n].view(np.uint32))
    assert np.array_equal(scene.Occlude(rays[:n]), occluded[:n])


# one part, then two, three and four, of equal and of unequal lengths
@pytest.mark.parametrize("n", [2 * PART - 1, 2 * PART, 2 * PART + 1, 3 * PART - 1,
                               3 * PART + 2, 4 * PART, MOST])
def test_parts_give_the_whole_calls_answers(made, n):
    check(made, n)


def test_behind_a_running_render(made):
    """The render's film and the query's rays and hits share the context's
    kept scratch."""
    import torch
    ctx, scene = made[:2]
    renderer = api.PTRenderer(api.PTRendererArgs(spp=64, max_bounces=8), seed=2)
    cam = scene.flat.camera
    want = renderer.Render(scene, cam).rgbw
    out = torch.zeros((512, 512, 4), device="cuda")
    for _ in range(2):
        out.zero_()
        torch.cuda.synchronize()
        renderer.render_device(scene, cam, out.data_ptr())
        check(made, 3 * PART + 2)
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))
