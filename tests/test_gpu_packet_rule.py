"""Waves large enough for bounce 0's packets (2 Mi paths, a packet within
half a triangle edge): single jobs and batches take them and render the
films a context without packets renders, bit for bit."""
import os

import numpy as np
import pytest

from ajisai_render_gb300 import api
from ajisai_render_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def context(packets):
    old = os.environ.get("AJG_PACKET_SHADOW")
    try:
        os.environ["AJG_PACKET_SHADOW"] = packets
        return api.Context(0)
    finally:
        if old is None:
            os.environ.pop("AJG_PACKET_SHADOW")
        else:
            os.environ["AJG_PACKET_SHADOW"] = old


def kinds(ctx, scene, camera, renderer):
    ctx.set_profiling(True)
    ctx.launch_log()
    renderer.Render(scene, camera)
    log = ctx.launch_log()
    ctx.set_profiling(False)
    return {r["kind"] for r in log}


def test_large_waves_take_packets_and_render_the_same():
    flats = [S.flatten(S.icosphere_scene(5, 2, 257, 190)), S.flatten(S.cornell_box(200, 230))]
    films = []
    for packets in ("0", "1"):
        ctx = context(packets)
        made = [api.GpuScene(ctx, f) for f in flats]
        big = [api.PTRenderer(api.PTRendererArgs(spp=48, max_bounces=3), seed=k) for k in (1, 2)]
        few = api.PTRenderer(api.PTRendererArgs(spp=4, max_bounces=3), seed=1)
        out = [r.Render(s, f.camera).rgbw for s, f, r in zip(made, flats, big)]
        out += [film.rgbw for film, _ in ctx.render_batch(
            [(s, f.camera, r) for s, f, r in zip(made, flats, big)] * 2)]
        films.append(out)
        if packets == "1":
            assert "any_packets" in kinds(ctx, made[0], flats[0].camera, big[0])
            assert "any_packets" not in kinds(ctx, made[0], flats[0].camera, few)
        ctx.close()
    for a, b in zip(*films):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    for a, b in zip(films[1][:2], films[1][2:]):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
