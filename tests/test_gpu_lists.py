"""The lists between the compositing kernels: a Gaussian's partial gradients gathered over its tiles."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import make_camera, random_model, rel_l2
from univeral_3d_reconstruction_system_b200.types import RasterSettings, TrainImage, TrainOptions

pytestmark = pytest.mark.gpu


def _close(u3dg, oracle, model, cam, st, w, rel):
    """Both backwards: over whole lists (the rasterizer's) and over segments (culled lists, the trainers')."""
    o = oracle.raster(1)
    o.forward(model, cam, st)
    og, ondc = o.backward(w)
    for culled in (True, False):
        r = u3dg.Rasterizer()
        r.set_tile_culling(culled)
        r.forward(model, cam, st)
        ndc = np.zeros(model.size(), np.float32)
        g = r.backward(model, w, None, ndc)
        for k in ("means", "scales", "quats", "opacities", "colors"):
            assert rel_l2(getattr(g, k), getattr(og, k)) <= rel, (k, culled)
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


def _stack(n, rng, opacity):
    """n Gaussians one behind the other, each over the whole of a small image."""
    m = random_model(n, rng, 0.05, 3.0, 0.5, 1.0)
    m.means[:, 2] = np.linspace(2.0, 4.0, n)
    m.opacities[:] = np.log(opacity / (1 - opacity))
    return m


@pytest.mark.parametrize("tile", [8, 16, 32])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 128, 129, 257, 700])
def test_backward_at_segment_edges(u3dg, oracle, n, tile):
    # Lists that end at, before and behind a segment's 64 (256 at tile 32) entries, blended to the end (no
    # pixel terminates: at most 700 alphas of 0.008) and over a background; some pixels terminate in a
    # second, opaque stack. Sums over 1,200 pixels: within 1e-4.
    rng = np.random.default_rng(n)
    w = rng.uniform(-1, 1, (37, 33, 3)).astype(np.float32)
    cam = make_camera(33, 37, 30.0)
    _close(u3dg, oracle, _stack(n, rng, 0.008), cam, RasterSettings(tile_size=tile, background=(0.3, 0.1, 0.2)), w, 1e-4)
    mixed = _stack(n, rng, 0.008)
    mixed.opacities[n // 2:] = 1.0
    mixed.scales[n // 2:] -= 3.0
    _close(u3dg, oracle, mixed, cam, RasterSettings(tile_size=tile), w, 1e-4)


@pytest.mark.parametrize("width, height, n", [(368, 400, 40), (480, 352, 40), (480, 352, 90)])
@pytest.mark.parametrize("background", [(0.0, 0.0, 0.0), (0.2, 0.4, 0.1)])
def test_backward_with_few_and_many_units(u3dg, oracle, width, height, n, background):
    # 575 blocks of 16x16 with one segment each (a unit per CTA at 592 CTAs and more), 660, and 660 with two.
    # Sums of up to 170,000 pixels in another order: 2^-24 sqrt(170,000) times a cancellation of 10 is 2.5e-4.
    rng = np.random.default_rng(n)
    w = rng.uniform(-1, 1, (height, width, 3)).astype(np.float32)
    _close(u3dg, oracle, _stack(n, rng, 0.05), make_camera(width, height, 1.5 * width), RasterSettings(background=background), w,
           3e-4)


@pytest.mark.parametrize("tile", [32, 64])
@pytest.mark.parametrize("width, height, n", [(368, 400, 40), (480, 352, 40), (480, 352, 700)])
def test_batch_depths_give_the_same_model(u3dg, tile, width, height, n):
    # On both sides of 592 units of the backward (4 per SM), where the order in which an entry's pixels are added
    # changes: 575, 660, and lists of more segments than one. The same bits.
    rng = np.random.default_rng(n)
    m = _stack(n, rng, 0.02)
    cam = make_camera(width, height, 1.5 * width)
    photo = TrainImage(cam, rng.integers(0, 256, (height, width, 3)).astype(np.uint8))
    flat = []
    for depth in (1, 2):
        t = u3dg.Trainer(m, [photo], 1.0, TrainOptions(max_gaussians=n, refine_stop=0, raster=RasterSettings(tile_size=tile)))
        t.set_raster_schedule(8, 1, depth)
        t.step(3)
        flat.append(t.model().flat())
    assert not np.array_equal(flat[0], m.flat())
    np.testing.assert_array_equal(flat[0], flat[1])


@pytest.mark.parametrize("culled", [False, True])
def test_a_non_finite_pixel_gradient_reaches_only_what_blends_there(u3dg, culled):
    rng = np.random.default_rng(3)
    m = random_model(200, rng, 1.0, 3.0, 0.02, 0.1)
    cam, st = make_camera(64, 48, 50.0), RasterSettings()
    w = rng.uniform(-1, 1, (48, 64, 3)).astype(np.float32)
    r = u3dg.Rasterizer()
    r.set_tile_culling(culled)
    r.forward(m, cam, st)
    clean = r.backward(m, w)
    w[20, 30, 1] = np.inf
    r.forward(m, cam, st)
    bad = r.backward(m, w)
    hit = ~np.isfinite(bad.opacities)
    # The Gaussians that blend at that pixel, found by the image's change when each is removed.
    base = r.forward(m, cam, st)[20, 30]
    blends = np.zeros(m.size(), bool)
    for i in range(m.size()):
        one = m.copy()
        one.opacities[i] = -30.0
        blends[i] = np.any(r.forward(one, cam, st)[20, 30] != base)
    assert 0 < blends.sum() < m.size() // 2
    assert np.all(hit <= blends)
    for k in ("means", "scales", "quats", "opacities", "colors"):
        a, b = getattr(bad, k)[~blends], getattr(clean, k)[~blends]
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("culled", [False, True])
@pytest.mark.parametrize("background", [(0.0, 0.0, 0.0), (0.2, 0.4, 0.1)])
def test_a_non_finite_colour_reaches_only_the_pixels_it_covers(u3dg, background, culled):
    rng = np.random.default_rng(4)
    m = random_model(120, rng, 1.0, 3.0, 0.02, 0.08)
    m.means[7] = [0.0, 0.0, 2.5]
    cam, st = make_camera(64, 48, 50.0), RasterSettings(background=background)
    w = rng.uniform(-1, 1, (48, 64, 3)).astype(np.float32)
    r = u3dg.Rasterizer()
    r.set_tile_culling(culled)
    clean_image = r.forward(m, cam, st)
    clean = r.backward(m, w)
    m.colors[7, 0] = np.inf
    image = r.forward(m, cam, st)
    bad = r.backward(m, w)
    covered = np.any(image != clean_image, axis=-1)
    assert 0 < covered.sum() < covered.size // 4
    # Gaussians none of whose pixels the coloured one covers keep their gradients.
    far = np.array([np.isfinite(bad.opacities[i]) for i in range(m.size())])
    assert far.sum() > 20
    same = [i for i in range(m.size()) if np.array_equal(bad.means[i], clean.means[i])]
    w0 = np.where(covered[..., None], 0.0, w).astype(np.float32)
    m.colors[7, 0] = 0.0
    r.forward(m, cam, st)
    masked = r.backward(m, w0)
    r.forward(m, cam, st)
    whole = r.backward(m, w)
    untouched = [i for i in range(m.size()) if np.array_equal(masked.opacities[i], whole.opacities[i])]
    assert untouched and set(untouched) - {7} <= set(same)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 64, 65, 129, 700])
@pytest.mark.parametrize("opacity", [0.008, 0.6])
def test_forward_kernels_agree_and_match_the_oracle(u3dg, oracle, n, opacity):
    # The left 256 columns of a 512x272 image (2,176 blocks of 8x8: one warp per block) and the same columns
    # as an image of their own (1,088 blocks: a team per block), with everything left of the optical axis
    # so that both project alike: the same bits, at lists around the batch sizes, ended by the cut-off or
    # not; and within 1e-5 of the oracle.
    rng = np.random.default_rng(n)
    m = _stack(n, rng, opacity)
    m.means[:, 0] = rng.uniform(-1.1, -0.35, n) * m.means[:, 2] * 0.5
    m.means[:, 1] = rng.uniform(-0.3, 0.3, n)
    m.scales -= 2.0
    wide = make_camera(512, 272, 480.0)
    left = make_camera(512, 272, 480.0)
    left.width = 256
    out = []
    for cam in (wide, left):
        r = u3dg.Rasterizer()
        image = r.forward(m, cam, RasterSettings(background=(0.1, 0.2, 0.3)))
        ft, nc = r.pixel_state()
        out.append([x.reshape(272, cam.width, -1)[:, :256] for x in (image, ft, nc)])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    assert out[0][2].max() > 0
    ref = oracle.render(m, left, RasterSettings(background=(0.1, 0.2, 0.3)))
    assert np.max(np.abs(out[1][0] - ref)) <= 1e-5


@pytest.mark.parametrize("n, tiles_x, tiles_y, wide", [(1, 1, 1, 1), (511, 3, 2, 2), (512, 5, 7, 3), (513, 64, 32, 5), (2049, 45, 45, 4),
                                                       (20_011, 64, 32, 3), (1500, 46, 45, 3), (700, 20, 15, 20)])
def test_tile_lists_at_chunk_and_path_edges(u3dg, oracle, n, tiles_x, tiles_y, wide):
    # Chunks of 512 ranks, their last rank and the next; exactly 2048 tiles (one tile per digit) and just
    # more (sorted by tile id); chunks with more intersections than they list (700 Gaussians in up to 300
    # tiles); equal depths; invisible Gaussians. Exact.
    rng = np.random.default_rng(n + tiles_x)
    depth = rng.choice(rng.uniform(0.5, 80.0, max(1, n // 3)).astype(np.float32), n)
    radius = (rng.random(n) < 0.9).astype(np.int32) * 7
    x0, y0 = rng.integers(0, tiles_x, n), rng.integers(0, tiles_y, n)
    x1 = np.minimum(tiles_x, x0 + 1 + rng.integers(0, wide, n))
    y1 = np.minimum(tiles_y, y0 + 1 + rng.integers(0, wide, n))
    rect = np.stack([x0, y0, x1, y1], 1).astype(np.int32)
    offsets, ids = u3dg.binTiles(depth, radius, rect, tiles_x, tiles_y)
    # Rasterizer.cpp:206-261: visible Gaussians by depth, ties by index, appended to each tile of their rect.
    lists = [[] for _ in range(tiles_x * tiles_y)]
    for i in np.argsort(depth, kind="stable"):
        if radius[i] > 0:
            for ty in range(y0[i], y1[i]):
                for tx in range(x0[i], x1[i]):
                    lists[ty * tiles_x + tx].append(i)
    np.testing.assert_array_equal(offsets, np.concatenate([[0], np.cumsum([len(x) for x in lists])]))
    np.testing.assert_array_equal(ids, np.concatenate([np.array(x, np.int32) for x in lists]) if len(ids) else ids)


@pytest.mark.parametrize("n", [1, 32, 33, 127, 128, 1025, 4095, 4096, 4097, 6145])
def test_depth_order_by_one_and_several_blocks(u3dg, n):
    # One kernel sorts up to 4096 Gaussians. Depths over many octaves, a third of them equal, a tenth of the
    # Gaussians invisible. Exact.
    rng = np.random.default_rng(n)
    depth = rng.choice(np.exp(rng.uniform(-8, 8, max(1, 2 * n // 3))).astype(np.float32), n)
    radius = (rng.random(n) < 0.9).astype(np.int32) * 3
    rect = np.tile(np.array([0, 0, 2, 1], np.int32), (n, 1))
    offsets, ids = u3dg.binTiles(depth, radius, rect, 2, 1)
    want = [i for i in np.argsort(depth, kind="stable") if radius[i] > 0]
    np.testing.assert_array_equal(offsets, [0, len(want), 2 * len(want)])
    np.testing.assert_array_equal(ids, np.array(want + want, np.int32))


@pytest.mark.parametrize("width, height, tile", [(240, 236, 16), (240, 240, 16), (235, 243, 16), (243, 235, 32), (235, 243, 64),
                                                 (350, 391, 8), (397, 405, 16)])
def test_tiles_in_order_of_their_lists(u3dg, oracle, width, height, tile):
    # On both sides of 888 blocks of 8x8, from which tiles are taken by descending list length, and with tiles
    # that reach over the image's edges; lists of 0 to 600 entries. Image within 1e-5, gradients as above.
    rng = np.random.default_rng(width)
    m = random_model(600, rng, 1.0, 3.0, 0.02, 0.3)
    m.means[:, 0] = np.abs(m.means[:, 0]) ** 2
    cam, st = make_camera(width, height, 0.8 * width), RasterSettings(tile_size=tile, background=(0.1, 0.2, 0.3))
    w = rng.uniform(-1, 1, (height, width, 3)).astype(np.float32)
    r = _close(u3dg, oracle, m, cam, st, w, 3e-4)
    np.testing.assert_allclose(r.forward(m, cam, st), oracle.raster(1).forward(m, cam, st), rtol=0, atol=1e-5)


def test_views_whose_lists_do_not_fit_at_first(u3dg):
    # 400 Gaussians over all of 4,800 tiles of 8x8: 1.9M intersections, above the first capacity of 2^20, between
    # views that fit. The bytes and the PSNR are those of views rendered one by one.
    rng = np.random.default_rng(8)
    m = _stack(400, rng, 0.1)
    m.scales += 2.0
    cams = [make_camera(w, h, 300.0) for w, h in ((64, 48), (640, 480), (640, 480), (97, 33), (640, 479))]
    st = RasterSettings(tile_size=8, background=(0.1, 0.2, 0.3))
    views = u3dg.renderViewsSh(m, None, 0, cams, st)
    r = u3dg.Rasterizer()
    images = [r.forward(m, c, st).reshape(c.height, c.width, 3) for c in cams]
    for view, image in zip(views, images):
        np.testing.assert_array_equal(view, TrainImage.quantize(image))
    photos = [TrainImage(c, rng.integers(0, 256, (c.height, c.width, 3)).astype(np.uint8)) for c in cams]
    t = u3dg.Trainer(m, photos, 1.0, TrainOptions(max_gaussians=400, raster=st))
    psnr = t.evaluatePsnr()
    want = []
    for p, image in zip(photos, images):
        d = image.astype(np.float64) - (p.rgb.astype(np.float32) * np.float32(1 / 255)).astype(np.float64)
        want.append(-10 * np.log10(np.mean(d * d)))
    assert abs(psnr - np.mean(want)) < 1e-5 * np.mean(want)


@pytest.mark.parametrize("width, height", [(161, 121), (1040, 800)])
@pytest.mark.parametrize("culled", [False, True])
@pytest.mark.parametrize("n", [0, 1, 32, 33, 513, 5000])
def test_backward_with_nothing_in_view(u3dg, n, culled, width, height):
    # Every Gaussian behind the camera, in a new rasterizer, in one that has seen them, and in one that has seen
    # fewer: no list has an entry (up to 2048 tiles and above), and every gradient is exactly zero.
    rng = np.random.default_rng(n)
    seen = random_model(n, rng, 1.0, 3.0, 0.02, 0.1)
    behind = seen.copy()
    behind.means[:, 2] = -behind.means[:, 2] - 10.0
    cam, st = make_camera(width, height, 0.8 * width), RasterSettings(background=(0.1, 0.2, 0.3))
    w = rng.uniform(-1, 1, (height, width, 3)).astype(np.float32)
    for before in (None, seen, random_model(max(1, n // 3), rng, 1.0, 3.0, 0.02, 0.1)):
        r = u3dg.Rasterizer()
        r.set_tile_culling(culled)
        if before is not None:
            r.forward(before, cam, st)
            r.backward(before, w)
        image = r.forward(behind, cam, st)
        np.testing.assert_array_equal(image, np.broadcast_to(np.float32(st.background), image.shape))
        ndc = np.zeros(n, np.float32)
        g = r.backward(behind, w, None, ndc)
        for k in ("means", "scales", "quats", "opacities", "colors"):
            assert not np.any(getattr(g, k)), k
        assert not np.any(ndc)
        offsets, ids = r.tiles()
        assert not np.any(offsets) and len(ids) == 0


@pytest.mark.parametrize("culled", [False, True])
@pytest.mark.parametrize("width, height", [(33, 37), (403, 340)])
@pytest.mark.parametrize("minimum", [float("nan"), -0.5, -2.0, float("-inf")])
def test_a_minimum_transmittance_that_nothing_is_below(u3dg, minimum, width, height, culled):
    # No pixel terminates, as with a minimum of 0: the same image and gradients, by a team per block and by one
    # warp (2,193 blocks of 8x8).
    rng = np.random.default_rng(width)
    m = _stack(90, rng, 0.3)
    m.scales -= 1.0
    cam = make_camera(width, height, 0.9 * width)
    w = rng.uniform(-1, 1, (height, width, 3)).astype(np.float32)
    out = []
    for least in (0.0, minimum):
        st = RasterSettings(background=(0.1, 0.2, 0.3), min_transmittance=least)
        r = u3dg.Rasterizer()
        r.set_tile_culling(culled)
        image = r.forward(m, cam, st)
        out.append([image, *r.pixel_state(), r.backward(m, w).flat()])
    assert out[0][2].max() == 90 and out[0][1].min() < 1e-4
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("culled", [False, True])
@pytest.mark.parametrize("background", [(0.0, 0.0, 0.0), (0.2, 0.4, 0.1)])
@pytest.mark.parametrize("colour, weight", [(2.0 ** 102, 2.0 ** 40), (2.0 ** 70, 2.0 ** 70), (2.0 ** 125, 16.0)])
def test_an_overflowing_product_reaches_only_what_blends_there(u3dg, colour, weight, background, culled):
    # A finite colour and a finite dL/dpixel whose product is infinite: Gaussians that blend at no pixel of the
    # bright one keep their gradients to the bit.
    rng = np.random.default_rng(6)
    m = random_model(150, rng, 1.0, 3.0, 0.02, 0.08)
    m.means[7] = [0.0, 0.0, 2.5]
    cam, st = make_camera(64, 48, 50.0), RasterSettings(background=background)
    w = (rng.uniform(0.5, 1, (48, 64, 3)) * weight).astype(np.float32)
    r = u3dg.Rasterizer()
    r.set_tile_culling(culled)
    image = r.forward(m, cam, st)
    clean = r.backward(m, w)
    bright = m.copy()
    bright.colors[7] = colour / 0.2820948
    covered = np.any(r.forward(bright, cam, st) != image, axis=-1)
    got = r.backward(bright, w)
    assert not np.isfinite(got.opacities[7])
    # Who blends at the covered pixels: whose opacity has a gradient from them.
    r.forward(m, cam, st)
    there = r.backward(m, np.repeat(covered[..., None], 3, axis=2).astype(np.float32))
    apart = there.opacities.reshape(-1) == 0
    assert apart.sum() > 50 and 0 < covered.sum() < covered.size // 4
    for k in ("means", "scales", "quats", "opacities", "colors"):
        np.testing.assert_array_equal(getattr(got, k)[apart], getattr(clean, k)[apart])


@pytest.mark.parametrize("n, tiles_x, tiles_y, wide", [(31, 4, 4, 2), (32, 7, 5, 3), (33, 64, 32, 64), (257, 64, 32, 64), (16_384, 13, 9, 3),
                                                       (16_385, 13, 9, 3), (17_001, 32, 24, 9)])
def test_tile_lists_of_few_and_many_gaussians(u3dg, n, tiles_x, tiles_y, wide):
    # Blocks of 32 ranks up to 16,384 Gaussians and of 512 beyond, with fewer and more intersections than a block
    # lists at a time. As above: exact.
    test_tile_lists_at_chunk_and_path_edges(u3dg, None, n, tiles_x, tiles_y, wide)


@pytest.mark.parametrize("n, size", [(40, 2.0), (700, 0.6), (17_000, 0.05)])
def test_culled_lists_of_large_gaussians(u3dg, n, size):
    # Rotated Gaussians over tens to hundreds of tiles of 8: a block of ranks lists its culled tiles in several
    # rounds. Every culled list is a subsequence of the whole one, nothing that blends is missing (same image and
    # transmittance, to the bit), and a Gaussian is in no tile twice.
    rng = np.random.default_rng(n)
    m = random_model(n, rng, 1.0, 3.0, 0.2 * size, size)
    m.scales[:, 1] -= 1.5
    cam, st = make_camera(320, 240, 300.0), RasterSettings(tile_size=8, background=(0.1, 0.2, 0.3))
    out = []
    for culled in (False, True):
        r = u3dg.Rasterizer()
        r.set_tile_culling(culled)
        out.append((r.forward(m, cam, st), r.pixel_state()[0], *r.tiles()))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    (_, _, whole, ids), (_, _, culled, some) = out
    assert len(some) < len(ids) and len(some) > 10_240
    for k in range(len(whole) - 1):
        full, part = ids[whole[k]:whole[k + 1]], some[culled[k]:culled[k + 1]]
        assert len(np.unique(part)) == len(part)
        place = {g: i for i, g in enumerate(full)}
        at = [place[g] for g in part]
        assert at == sorted(at)


@pytest.mark.parametrize("width, height", [(312, 304), (312, 312)])
@pytest.mark.parametrize("background", [(0.0, 0.0, 0.0), (0.2, 0.4, 0.1)])
def test_training_with_either_backward_at_tile_8(u3dg, oracle, width, height, background):
    # 1,482 and 1,521 tiles of 8, on both sides of the 1,500 beyond which the trainers replay whole lists: five steps
    # agree with the oracle's trainer, as trainings in another order of summation do.
    rng = np.random.default_rng(width + height)
    m = random_model(600, rng, 1.0, 3.0, 0.05, 0.3)
    cam = make_camera(width, height, 0.9 * width)
    photos = [TrainImage(cam, rng.integers(0, 256, (height, width, 3)).astype(np.uint8))]
    opt = TrainOptions(max_gaussians=600, refine_stop=0, raster=RasterSettings(tile_size=8, background=background))
    t, o = u3dg.Trainer(m, photos, 1.0, opt), oracle.trainer(m, photos, 1.0, opt, threads=4)
    t.step(5)
    o.step(5)
    a, b = t.stats(), o.stats()
    assert abs(a.loss - b.loss) <= 1e-4 * abs(b.loss) and abs(a.psnr - b.psnr) <= 1e-3
    for k in ("means", "scales", "quats", "opacities", "colors"):
        assert rel_l2(getattr(t.model(), k), getattr(o.model(), k)) < 1e-3, k


@pytest.mark.parametrize("n", [1, 7, 8, 9, 16, 31, 32, 33, 40, 64])
def test_partial_sums_at_chunk_edges(u3dg, oracle, n):
    # Every Gaussian in four tiles of 16: 4 to 256 entries, 128 (four chunks of 32) to 32 ranks. Sums over 1,024
    # pixels: within 1e-4.
    rng = np.random.default_rng(n)
    m = random_model(n, rng, 0.01, 3.0, 0.05, 0.1)
    m.means[:, 2] = np.linspace(2.9, 3.1, n)
    cam = make_camera(32, 32, 40.0)
    cam.cx = cam.cy = 15.5
    w = rng.uniform(-1, 1, (32, 32, 3)).astype(np.float32)
    r = _close(u3dg, oracle, m, cam, RasterSettings(background=(0.1, 0.2, 0.3)), w, 1e-4)
    r.set_tile_culling(False)
    r.forward(m, cam, RasterSettings())
    assert len(r.tiles()[1]) == 4 * n


@pytest.mark.parametrize("tile", [8, 16, 64])
@pytest.mark.parametrize("n, hidden", [(1, 32_768), (7, 32_768), (8, 32_768), (9, 32_768), (33, 32_768), (32_700, 69)])
def test_few_and_many_gaussians_are_updated_alike(u3dg, n, hidden, tile):
    # The chain rule takes 8 Gaussians to a warp up to 32,768 and 32 beyond: n Gaussians, and the same ones with so
    # many more that no view sees. The same model, to the bit.
    rng = np.random.default_rng(n)
    m = random_model(n, rng, 1.0, 3.0, 0.03, 0.4 if n < 100 else 0.05)
    far = random_model(1, rng, 1.0, 3.0, 0.05, 0.1)
    far.means[:] = (0.0, 0.0, -9.0)
    cam = make_camera(128, 96, 110.0)
    photo = TrainImage(cam, rng.integers(0, 256, (96, 128, 3)).astype(np.uint8))
    both = m.copy()
    for k in ("means", "scales", "quats", "opacities", "colors"):
        setattr(both, k, np.concatenate([getattr(m, k), np.repeat(getattr(far, k), hidden, axis=0)]))
    out = []
    for model in (m, both):
        t = u3dg.Trainer(model, [photo], 1.0, TrainOptions(max_gaussians=model.size(), refine_stop=0, raster=RasterSettings(tile_size=tile)))
        t.step(4)
        out.append(t.model())
    assert not np.array_equal(out[0].colors, m.colors)
    for k in ("means", "scales", "quats", "opacities", "colors"):
        np.testing.assert_array_equal(getattr(out[0], k), getattr(out[1], k)[:n], err_msg=k)
