"""The lists between the compositing kernels: a Gaussian's partial gradients gathered over its tiles."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import make_camera, random_model, rel_l2
from univeral_3d_reconstruction_system_b200.types import RasterSettings

pytestmark = pytest.mark.gpu


def _close(u3dg, oracle, model, cam, st, w, rel):
    r = u3dg.Rasterizer()
    r.forward(model, cam, st)
    ndc = np.zeros(model.size(), np.float32)
    g = r.backward(model, w, None, ndc)
    o = oracle.raster(1)
    o.forward(model, cam, st)
    og, ondc = o.backward(w)
    for k in ("means", "scales", "quats", "opacities", "colors"):
        assert rel_l2(getattr(g, k), getattr(og, k)) <= rel, k
    assert rel_l2(ndc, ondc) <= rel
    return r


@pytest.mark.parametrize("width, height, tile", [(16, 16, 16), (128, 64, 16), (132, 64, 16), (320, 176, 16), (320, 176, 8),
                                                 (160, 96, 32)])
def test_gaussians_in_few_and_many_tiles(u3dg, oracle, width, height, tile):
    # Gaussians larger than the image beside small ones: 1, 32, 36, 220 and 880 tiles each, on both sides
    # of the tile count above which a warp adds one Gaussian together, and several blocks per tile.
    # Sums of up to 56,000 pixels in another order: 2^-24 sqrt(56,000) times a cancellation of 10 is 1.4e-4.
    rng = np.random.default_rng(width)
    small, large = random_model(150, rng, 1.0, 3.0, 0.02, 0.1), random_model(5, rng, 0.5, 3.5, 3.0, 6.0)
    for k in ("means", "scales", "quats", "opacities", "colors"):
        setattr(small, k, np.concatenate([getattr(small, k), getattr(large, k)]))
    cam = make_camera(width, height, 0.8 * width)
    w = rng.uniform(-1, 1, (height, width, 3)).astype(np.float32)
    _close(u3dg, oracle, small, cam, RasterSettings(tile_size=tile, background=(0.1, 0.2, 0.3)), w, 2e-4)
