"""Trainers on a device that is nearly full: they do without the backward's segments, half of what an intersection
takes, before they refuse."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from helpers import make_camera, random_model, rel_l2
from univeral_3d_reconstruction_system_b200.types import RasterSettings, TrainImage, TrainOptions

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.fixture
def fill():
    """fill(bytes): takes all device memory but so much, until the test ends."""
    import torch

    held = []

    def take(left):
        torch.cuda.empty_cache()
        held.append(torch.empty(max(0, torch.cuda.mem_get_info()[0] - int(left)), dtype=torch.uint8, device="cuda"))

    yield take
    held.clear()
    torch.cuda.empty_cache()


def _free():
    import torch

    return torch.cuda.mem_get_info()[0]


def _scene(tile, cap, seed=0):
    rng = np.random.default_rng(seed)
    m = random_model(2000, rng, 1.0, 3.0, 0.02, 0.1)
    cam = make_camera(96, 72, 80.0)
    photos = [TrainImage(dataclasses.replace(cam, cx=cam.cx + d), rng.integers(0, 256, (72, 96, 3)).astype(np.uint8))
              for d in (-9.0, 0.0, 7.0)]
    return m, photos, 1.0, TrainOptions(max_gaussians=cap, refine_stop=0, raster=RasterSettings(tile_size=tile))


def _same_training(a, b):
    # The order in which a Gaussian's gradient is summed differs (as with tile culling on and off).
    assert abs(a.evaluatePsnr() - b.evaluatePsnr()) < 0.02
    for k in ("means", "scales", "quats", "opacities", "colors"):
        assert rel_l2(getattr(a.model(), k), getattr(b.model(), k)) < 1e-2, k


@pytest.mark.parametrize("tile", [8, 16, 32])
def test_a_trainer_that_would_not_fit_with_segments(u3dg, fill, tile):
    cap = 1_000_000 if tile == 8 else 400_000
    free = _free()
    a = u3dg.Trainer(*_scene(tile, cap))
    full = free - _free()
    a.step(33)  # single steps and graph runs
    fill(full - 150 * MB)
    b = u3dg.Trainer(*_scene(tile, cap))
    assert b.evaluatePsnr() > 0
    b.step(33)
    assert b.graph_launches() > 0
    _same_training(a, b)


def test_a_trainer_whose_lists_outgrow_the_device(u3dg, fill):
    # 1,100 Gaussians over all of 1,200 tiles: 1.3M intersections, above the first capacity of 2^20. Room for the
    # larger lists and partials (100 MB), not for their segments (another 106).
    rng = np.random.default_rng(1)
    m = random_model(1100, rng, 0.05, 3.0, 0.5, 1.0)
    m.means[:, 2] = np.linspace(2.0, 4.0, 1100)
    m.scales += 2.0
    m.opacities[:] = -4.0
    cam = make_camera(640, 480, 300.0)
    scene = (m, [TrainImage(cam, rng.integers(0, 256, (480, 640, 3)).astype(np.uint8))], 1.0,
             TrainOptions(max_gaussians=1100, refine_stop=0))
    a = u3dg.Trainer(*scene)
    a.step(15)
    assert a.replays() >= 1
    b = u3dg.Trainer(*scene)
    fill(150 * MB)
    b.step(15)
    assert b.replays() >= 1
    _same_training(a, b)


def test_a_batch_that_would_not_fit_with_segments(u3dg, fill):
    scenes = [_scene(16, 400_000, s) for s in range(3)]
    free = _free()
    one = u3dg.Trainer(*scenes[0])
    full = free - _free()
    one.step(23)
    fill(2.4 * full)  # two trainers with segments and 0.4 of one, or three without
    b = u3dg.Batch(scenes, autotune=False)
    b.step(23)
    _same_training(one, b.trainer(0))
    b.close()


def test_no_backward_after_a_forward_that_ran_out_of_memory(u3dg, fill):
    rng = np.random.default_rng(2)
    m = random_model(500, rng, 1.0, 3.0, 0.02, 0.1)
    cam, st = make_camera(96, 72, 80.0), RasterSettings()
    w = rng.uniform(-1, 1, (72, 96, 3)).astype(np.float32)
    r = u3dg.Rasterizer()
    r.forward(m, cam, st)
    want = r.backward(m, w)
    large = m.copy()
    for k in ("means", "scales", "quats", "opacities", "colors"):
        setattr(large, k, np.tile(getattr(m, k), (4000,) + (1,) * (getattr(m, k).ndim - 1)))
    fill(200 * MB)  # 2M Gaussians take 1.5 GB of lists
    with pytest.raises(u3dg.U3dgError, match="memory"):
        r.forward(large, cam, st)
    for model in (large, m):
        with pytest.raises(u3dg.U3dgError):
            r.backward(model, w)
    r.forward(m, cam, st)
    np.testing.assert_array_equal(r.backward(m, w).flat(), want.flat())
