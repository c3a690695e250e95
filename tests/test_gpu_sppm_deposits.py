"""SPPM's deposits: the photon records joined with the visible points entry
by entry, against the oracle's per-photon walk."""
import numpy as np
import pytest

from ajisai_render_gb300 import api
from ajisai_render_gb300 import scenes as S
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def radiance(args, wave_paths=0, seed=5, size=(40, 24)):
    flat = S.flatten(S.cornell_area(*size))
    ctx = api.Context(0, wave_paths=wave_paths)
    try:
        return flat, api.SPPMRenderer(args, seed).RenderRadiance(api.GpuScene(ctx, flat),
                                                                 flat.camera)
    finally:
        ctx.close()


# radii from less than a pixel to the whole box in one cell (every visible
# point and photon under a few entries); photon counts around the join's
# tiles of 32 and a depth without any deposit
@pytest.mark.parametrize("radius,photons,depth", [
    (0.004, 3001, 6), (0.05, 33, 6), (0.3, 1000, 4), (2.0, 2047, 3), (0.05, 1, 10),
    (0.05, 500, 1), (0.05, 500, 0)])
def test_deposits_match_the_oracle(radius, photons, depth):
    args = api.SPPMRendererArgs(forward_max_depth=5, init_radius=radius, iteration_count=3,
                                photons_per_iteration=photons, photon_min_depth=2,
                                photon_max_depth=depth)
    flat, rad = radiance(args)
    ref, _ = O.OracleScene(flat, search_radius=14).sppm(
        flat.camera, dict(iterations=3, photons_per_iteration=photons, forward_max_depth=5,
                          photon_min_depth=2, photon_max_depth=depth, init_radius=radius),
        seed=5)
    # a photon whose path a last-ulp difference turns elsewhere moves the
    # pixels it lands in, as in the parity tests: within 1e-3 on 97% of the
    # pixels, or with few photons on all but what two of them can reach
    close = np.isclose(rad, ref, rtol=1e-3, atol=1e-5, equal_nan=True).all(-1)
    assert close.mean() > 0.97, close.mean()


def test_chunks_sum_to_the_same_estimate():
    """1,024 photons a chunk or all in one: the same deposits, summed in
    another order (up to some hundred float32 terms a pixel)."""
    args = api.SPPMRendererArgs(forward_max_depth=5, init_radius=0.08, iteration_count=2,
                                photons_per_iteration=10_007, photon_max_depth=6)
    _, a = radiance(args)
    _, b = radiance(args, wave_paths=1024)
    np.testing.assert_allclose(b, a, rtol=1e-4, atol=1e-6, equal_nan=True)


def test_waves_of_iterations_sum_to_the_same_estimate():
    """70 iterations of 31,000 photons (several waves of many iterations, the
    last one short) and the same in a context whose waves hold one iteration
    or a part of it."""
    args = api.SPPMRendererArgs(forward_max_depth=4, init_radius=0.05, iteration_count=70,
                                photons_per_iteration=31_000, photon_max_depth=5)
    _, a = radiance(args)
    _, b = radiance(args, wave_paths=40_960)
    _, c = radiance(args, wave_paths=16_384)
    np.testing.assert_allclose(b, a, rtol=1e-4, atol=1e-6, equal_nan=True)
    np.testing.assert_allclose(c, a, rtol=1e-4, atol=1e-6, equal_nan=True)
