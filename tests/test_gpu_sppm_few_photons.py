"""SPPM with a few photons whose deposits each cover a large share of the film:
which pixels received photon energy, and how much, as the oracle's per-photon
walk has it."""
import numpy as np
import pytest

from ajisai_render_gb300 import api
from ajisai_render_gb300 import scenes as S
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def photon_part(render, photons, iterations, radius):
    """The radiance with deposits less that without (a photon deposits from
    depth 2 on)."""
    args = dict(iterations=iterations, photons_per_iteration=photons, forward_max_depth=5,
                photon_min_depth=2, init_radius=radius)
    return (render(dict(args, photon_max_depth=10))
            - render(dict(args, photon_max_depth=1)))


@pytest.mark.parametrize("photons,iterations,radius", [
    (1, 16, 0.4), (2, 8, 0.6), (31, 1, 0.3), (33, 2, 2.0)])
def test_photon_energy_matches_the_oracle(photons, iterations, radius):
    flat = S.flatten(S.cornell_area(40, 24))
    ctx = api.Context(0)
    scene = api.GpuScene(ctx, flat)

    def gpu(p):
        a = api.SPPMRendererArgs(
            forward_max_depth=p["forward_max_depth"], init_radius=p["init_radius"],
            iteration_count=p["iterations"],
            photons_per_iteration=p["photons_per_iteration"],
            photon_min_depth=p["photon_min_depth"], photon_max_depth=p["photon_max_depth"])
        return api.SPPMRenderer(a, 5).RenderRadiance(scene, flat.camera)

    got = photon_part(gpu, photons, iterations, radius)
    oracle = O.OracleScene(flat, search_radius=14)
    want = photon_part(lambda p: oracle.sppm(flat.camera, p, seed=5)[0], photons,
                       iterations, radius)
    ctx.close()
    finite = np.isfinite(want).all(-1)
    assert np.array_equal(np.isfinite(got).all(-1), finite)
    got, want = got[finite], want[finite]
    lit = (want != 0).any(-1)
    assert lit.mean() > 0.1
    # a point at the rim of a deposit's radius may fall on either side of it
    assert ((got != 0).any(-1) != lit).sum() <= 4
    # a dropped or doubled deposit moves the sum by its share, some percent
    np.testing.assert_allclose(got.sum(0), want.sum(0), rtol=2e-3)
