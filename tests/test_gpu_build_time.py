"""ajg_scene_info.build_ms is the build's GPU time: copies from host memory that
was never touched before, which hold the host far longer, are not in it."""
import numpy as np
import pytest

from ajisai_render_gb300 import api
from ajisai_render_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def test_build_ms_leaves_out_the_copies():
    ctx = api.Context(0)
    n = 6_000_000
    rng = np.random.default_rng(3)
    t = (rng.uniform(0, 1, (n, 1, 3)) + rng.normal(0, 0.003, (n, 3, 3))).astype(np.float32)
    t = t.reshape(n, 9)
    world = np.array([-1, -1, -1, 2, 2, 2], np.float32)
    mats = S.Diffuse((0.5, 0.5, 0.5)).pack()[None]

    def build_ms(corner, mat, flags):
        flat = S.FlatScene(t, corner, mat, flags, world, mats, np.zeros((0, 12), np.float32), None)
        scene = api.GpuScene(ctx, flat)
        ms = scene.info()["build_ms"]
        scene.release()
        return ms

    # AJG_MESH_HAS_NORMALS: the corner normals are copied in
    mat, flags = np.zeros(n, np.int32), np.full(n, 4, np.int32)
    corner = np.ones((n, 9), np.float32)
    build_ms(corner, mat, flags)
    again = min(build_ms(corner, mat, flags) for _ in range(3))
    # np.zeros: pages the copy is the first to touch
    fresh = max(build_ms(np.zeros((n, 9), np.float32), mat, flags) for _ in range(4))
    ctx.close()
    assert fresh < 1.5 * again, (fresh, again)
