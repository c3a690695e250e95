"""The PLOC build's limit of 100,000 iterations, at inputs that need one
iteration more or just as many."""
import numpy as np
import pytest

from ajisai_render_gb300 import _lib, api
from ajisai_render_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def make(ctx, n):
    """n equal triangles: they merge a pair an iteration, n - 1 in all."""
    tris = np.tile(np.array([[0, 0, 0, 1, 0, 0, 0, 1, 0]], np.float32), (n, 1))
    flat = S.FlatScene(tris, np.zeros((n, 9), np.float32), np.zeros(n, np.int32),
                       np.zeros(n, np.int32), np.array([0, 0, 0, 1, 1, 1], np.float32),
                       S.Diffuse((0.5, 0.5, 0.5)).pack()[None],
                       np.zeros((0, 12), np.float32), None)
    return api.GpuScene(ctx, flat, api.CreatePLOCAggregate(2))


def test_the_limit():
    ctx = api.Context(0)
    with pytest.raises(_lib.AjgError, match="did not converge"):
        make(ctx, 100_002)
    assert make(ctx, 100_001).info()["ploc_iterations"] == 100_000
    ctx.close()
