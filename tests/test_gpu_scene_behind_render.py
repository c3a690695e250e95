"""A scene made behind an asynchronous render of the same context: both use the
context's kept scratch, so the scene's copies must wait for the render."""
import numpy as np
import pytest

from ajisai_render_gb300 import api
from ajisai_render_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def pinned(flat):
    """The flat scene with its arrays in pinned memory (copies that return at
    once)."""
    import torch
    arrays = {k: torch.from_numpy(np.ascontiguousarray(getattr(flat, k))).pin_memory()
              for k in ("tris", "corner_n", "tri_mat", "tri_flags")}
    for k, t in arrays.items():
        setattr(flat, k, t.numpy())
    return flat, arrays


@pytest.mark.parametrize("where", ["pageable", "pinned"])
@pytest.mark.parametrize("subdiv", [2, 5])
def test_render_and_scene_behind_it_are_unchanged(where, subdiv):
    import torch
    ctx = api.Context(0)
    first = api.GpuScene(ctx, S.flatten(S.icosphere_scene(5, 2, 1024, 1024)))
    cam = first.flat.camera
    renderer = api.PTRenderer(api.PTRendererArgs(spp=16, max_bounces=8), seed=3)
    small = api.PTRenderer(api.PTRendererArgs(spp=4, max_bounces=4), seed=4)
    flat = S.flatten(S.icosphere_scene(subdiv, 7, 64, 48))
    if where == "pinned":
        flat, keep = pinned(flat)
    # a larger film first: the kept scratch then holds the scene's temporaries
    renderer.Render(first, S.flatten(S.icosphere_scene(1, 2, 1280, 1024)).camera)

    def film():
        out = torch.zeros((1024, 1024, 4), device="cuda")
        torch.cuda.synchronize()
        renderer.render_device(first, cam, out.data_ptr())
        return out

    want = film()
    torch.cuda.synchronize()
    alone = small.Render(api.GpuScene(ctx, flat), flat.camera).rgbw
    for _ in range(3):
        got = film()
        scene = api.GpuScene(ctx, flat)  # the render is still running
        behind = small.Render(scene, flat.camera).rgbw
        torch.cuda.synchronize()
        assert np.array_equal(got.cpu().numpy().view(np.uint32),
                              want.cpu().numpy().view(np.uint32))
        assert np.array_equal(behind.view(np.uint32), alone.view(np.uint32))
        scene.release()
    ctx.close()
