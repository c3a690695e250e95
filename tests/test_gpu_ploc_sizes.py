"""The PLOC build around the sizes its kernels change at: the one-block tail
(1,024 clusters), tiles of 256 and 1,024, small and large sorts, search radii
beyond a tile, and inputs that merge one pair an iteration."""
import numpy as np
import pytest

from ajisai_render_gb300 import api
from ajisai_render_gb300 import scenes as S
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


def soup(n, seed=0, same=False):
    rng = np.random.default_rng(seed)
    c = rng.uniform(0, 1, (1 if same else n, 1, 3))
    t = (c + rng.normal(0, 0.02, (1 if same else n, 3, 3))).reshape(-1, 9)
    return np.repeat(t, n, 0).astype(np.float32) if same else t.astype(np.float32)


def check(ctx, tris, radius, width=0):
    world = np.concatenate([tris.reshape(-1, 3).min(0), tris.reshape(-1, 3).max(0)])
    n = len(tris)
    flat = S.FlatScene(tris, np.zeros((n, 9), np.float32), np.zeros(n, np.int32),
                       np.zeros(n, np.int32), world.astype(np.float32),
                       S.Diffuse((0.5, 0.5, 0.5)).pack()[None],
                       np.zeros((0, 12), np.float32), None)
    sc = api.GpuScene(ctx, flat, api.CreatePLOCAggregate(radius, bvh_width=width))
    nb, ncf, perm = sc.download_bvh()
    onb, oncf, operm = O.ploc_build(tris, flat.world, radius)
    assert np.array_equal(perm, operm)
    assert np.array_equal(ncf, oncf)
    assert np.array_equal(nb.view(np.uint32), onb.view(np.uint32))
    # and the collapsed layouts hold every triangle: rays at their centres
    m = min(n, 500)
    a = tris.reshape(n, 3, 3)[:m].mean(1)
    d = np.cross(tris[:m, 3:6] - tris[:m, 0:3], tris[:m, 6:9] - tris[:m, 0:3])
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.concatenate([a + 0.01 * d, -d, np.full((m, 1), 1e-6),
                           np.full((m, 1), np.inf)], 1).astype(np.float32)
    t, p, u, v = sc.Intersect(rays)
    ot, op, _, _ = O.trace(tris, rays)[:4]
    assert np.array_equal(p, op) and np.array_equal(t, ot)


@pytest.mark.parametrize("n,radius", [
    (1, 14), (2, 1), (3, 14), (255, 16), (1023, 16), (1024, 16), (1025, 16), (1026, 1),
    (1281, 300), (4097, 16), (5000, 1024), (262_144, 8), (262_145, 8)])
def test_sizes_match_the_oracle(ctx, n, radius):
    check(ctx, soup(n, n), radius)


@pytest.mark.parametrize("width", [2, 8, 0x104])
def test_other_layouts_match_the_oracle(ctx, width):
    check(ctx, soup(3001, 5), 14, width)


def test_one_pair_an_iteration(ctx):
    """Equal triangles: the first minimum in index order pairs only the
    first two clusters, so the build takes an iteration per triangle."""
    check(ctx, soup(1200, 1, same=True), 14)
