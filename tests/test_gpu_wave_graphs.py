"""The request loop's waves, launched as they are and as captured graphs: a
kind of wave is captured when it has come back, and renders the same bits."""
import numpy as np
import pytest

from ajisai_render_gb300 import api
from ajisai_render_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def test_repeated_waves_are_captured_and_render_the_same():
    ctx = api.Context(0)
    made = [api.GpuScene(ctx, S.flatten(make(61, 43)))
            for make in (S.cornell_box, S.cornell_area, S.material_box)]
    renderer = api.PTRenderer(api.PTRendererArgs(spp=3, max_bounces=6), seed=9)
    # the scene with the most lights first: the arena then stays as it is
    made.sort(key=lambda s: -s.flat.emit_info.shape[0] - s.flat.lights.shape[0])
    films, builds = [], []
    for _ in range(5):
        films.append([ctx.render_batch([(s, s.flat.camera, renderer)])[0][0].rgbw
                      for s in made])
        builds.append(ctx.serve_stats()["graph_builds"])
    ctx.close()
    for later in films[1:]:
        for a, b in zip(films[0], later):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    # no capture for what has come once, and none twice
    assert builds[0] == 0 and builds[-1] == builds[-2] > 0
