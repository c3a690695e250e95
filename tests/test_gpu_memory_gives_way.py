"""Where device memory is short, the scratch a context keeps between its calls
is given back: what fits without it succeeds."""
import numpy as np
import pytest

from ajisai_render_gb300 import api
from ajisai_render_gb300 import scenes as S

pytestmark = pytest.mark.gpu

MB = 1 << 20


class Filled:
    """All device memory taken but `left` bytes."""

    def __init__(self, left):
        import torch
        torch.cuda.empty_cache()
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        self.block = torch.empty(free - left, dtype=torch.uint8, device="cuda")

    def release(self):
        import torch
        self.block = None
        torch.cuda.empty_cache()


def fill_scratch(ctx, scene, camera):
    """A call whose scratch takes over 1 GB (kept up to 4 GB)."""
    api.SPPMRenderer(api.SPPMRendererArgs(iteration_count=1, photons_per_iteration=2_000_000,
                                          init_radius=0.01), 1).Render(scene, camera)


def test_a_jobs_film():
    ctx = api.Context(0)
    flat = S.flatten(S.cornell_area(32, 32))
    scene = api.GpuScene(ctx, flat)
    renderer = api.PTRenderer(api.PTRendererArgs(spp=1, max_bounces=1), seed=1)
    camera = S.flatten(S.cornell_area(4096, 4096)).camera
    # the loop's arena and kernels, and the film's pixels without a limit
    want = ctx.render_batch([(scene, camera, renderer)])[0][0].rgbw
    fill_scratch(ctx, scene, flat.camera)
    fill = Filled(600 * MB)  # film and result take 805 MB
    try:
        film, status = ctx.render_batch([(scene, camera, renderer)])[0]
    finally:
        fill.release()
    ctx.close()
    assert status["state_name"] == "done"
    assert np.array_equal(film.rgbw.view(np.uint32), want.view(np.uint32))


def test_a_scenes_collapsed_tree():
    """327,682 triangles: 76 MB of arrays, then a tree of some 17 MB while the
    build's 109 MB of temporaries are in the kept scratch."""
    ctx = api.Context(0)
    flat = S.flatten(S.cornell_area(32, 32))
    big = S.flatten(S.icosphere_scene(7, 1, 64, 64))
    scene = api.GpuScene(ctx, flat)
    rays = np.tile(np.array([[0.3, 3, 0.2, 0, -1, 0, 1e-4, np.inf]], np.float32), (8, 1))
    made = api.GpuScene(ctx, big)
    want = made.Intersect(rays)
    made.release()
    for left in range(78, 102, 4):
        fill_scratch(ctx, scene, flat.camera)
        fill = Filled(left * MB)
        try:
            made = api.GpuScene(ctx, big)
        finally:
            fill.release()
        for a, b in zip(made.Intersect(rays), want):
            assert np.array_equal(a, b)
        made.release()
    ctx.close()
