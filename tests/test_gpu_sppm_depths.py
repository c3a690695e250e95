"""SPPM with a depth limit whose deposits do not fit the record buffer at
once: they are joined with the visible points every few depths."""
import numpy as np
import pytest

from ajisai_render_gb300 import api
from ajisai_render_gb300 import scenes as S

pytestmark = pytest.mark.gpu


# 2^25 records: joined after 111, 11 and 2 depths of 127, 39 and 5; the short
# waves' chunks hold all depths
@pytest.mark.parametrize("photons,depth,short", [
    (300_000, 128, 65_536), (3_000_000, 40, 262_144), (12_000_000, 6, 1 << 20)])
def test_joins_every_few_depths_sum_to_the_same_estimate(photons, depth, short):
    flat = S.flatten(S.cornell_area(40, 24))
    args = api.SPPMRendererArgs(forward_max_depth=4, init_radius=0.01, iteration_count=2,
                                photons_per_iteration=photons, photon_min_depth=5,
                                photon_max_depth=depth, photon_cont_prob=0.95)
    out = []
    for wave_paths in (0, short):
        ctx = api.Context(0, wave_paths=wave_paths)
        out.append(api.SPPMRenderer(args, 5).RenderRadiance(api.GpuScene(ctx, flat),
                                                           flat.camera))
        ctx.close()
    # the same deposits summed in another order: terms of one sign, at most
    # some thousand a pixel and iteration, 1.2e-7 each
    np.testing.assert_allclose(out[0], out[1], rtol=5e-4, atol=1e-6, equal_nan=True)
