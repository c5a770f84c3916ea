"""The rasters at the sizes where they can go wrong, against the oracle's
raster of the same lists: the stage raster in reference mode on hand-made
tile lists (batch remainders, image sizes that cut tiles, every tile shape,
entries whose exponent is not a number) and the record raster of whole T_min
frames."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTS = (0, 1, 31, 32, 33, 63, 64, 65, 96, 130)


def _lists(rng, tiles, n):
    counts = [COUNTS[t % len(COUNTS)] for t in range(tiles)]
    ends = np.cumsum(counts)
    ranges = np.stack([ends - counts, ends], 1).astype(np.int32)
    return ranges, rng.integers(0, n, max(int(ends[-1]), 1)).astype(np.int32)


@pytest.mark.parametrize("tile", [(16, 16), (16, 8), (8, 8)])
@pytest.mark.parametrize("size", [(1, 1), (17, 9), (47, 33), (64, 48), (250, 131), (1201, 651)])
@pytest.mark.parametrize("wild", [False, True])
def test_reference_raster(gs, O, tile, size, wild):
    import torch
    rng = np.random.default_rng(size[0] * 7 + tile[1])
    W, H = size
    rc = gs.RenderConfig.reference()
    rc.tile_w, rc.tile_h = tile
    cam = gs.look_at((0, 0, 3.0), (0, 0, 0), (0, 1, 0), 60.0, W, H, 0.1, 100.0)
    tiles, n = gs.num_tiles(W, H, rc), 400
    ranges, vals = _lists(rng, tiles, n)
    xy = rng.uniform(-1, 1, (n, 2)).astype(np.float32)
    conic = np.zeros((n, 4), np.float32)
    conic[:, 0], conic[:, 2] = rng.uniform(1, 40, (2, n))
    conic[:, 1] = rng.uniform(-0.9, 0.9, n) * np.sqrt(conic[:, 0] * conic[:, 2])
    # 130 entries of opacity 0.02 leave T above 0.07: the 0.02 test never decides
    color = np.concatenate([rng.uniform(0, 1, (n, 3)), rng.uniform(0, 0.02, (n, 1))], 1).astype(np.float32)
    if wild:
        # not a number or infinite: saturate(NaN) = 0, exp(+inf) saturates, exp(-inf) = 0
        conic[0::40, 0] = np.nan
        conic[1::40, 2] = np.inf
        conic[2::40, 0], conic[2::40, 1] = np.inf, -np.inf
        conic[3::40, 0] = -np.inf
        conic[4::40, 0] = 3e38
        xy[5::40, 1] = np.nan
        conic[6::40, :3] = -1.0
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    img = torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda")
    gs.stage_raster(cam, rc, dev(ranges), dev(vals), dev(xy), dev(conic), dev(color), img)
    ref = O.raster(cam, rc, ranges, vals, xy, conic, color)
    # |q| <= 600, so a last-bit difference of q or of the pixel's centre moves
    # a density by at most 1e-4 of itself and a colour by less than one step;
    # one more for the truncation to 8 bits
    diff = np.abs(img.cpu().numpy().astype(int) - ref.astype(int))
    assert diff.max() <= 1, diff.max()


@pytest.mark.parametrize("tile", [(16, 16), (16, 8), (8, 8)])
@pytest.mark.parametrize("chunk", [32, 64])
@pytest.mark.parametrize("n,size", [(1, (9, 5)), (40, (17, 16)), (700, (33, 47)), (9000, (50, 31)), (9000, (1201, 651))])
def test_record_raster(gs, O, tile, chunk, n, size):
    """Whole T_min frames whose blocks are cut by the image's edges, with one
    entry up to a few thousand per tile, against the oracle's raster of the
    frame's own lists and projected floats."""
    import torch
    W, H = size
    sc = gs.scenes.uniform_scene(n, seed=n, log_scale_mu=-2.5 if W < 100 else -4.0)
    rc = gs.RenderConfig(tile_w=tile[0], tile_h=tile[1], raster_chunk=chunk)
    cam = gs.look_at((0.1, 0.2, 3.0), (0, 0, 0), (0, 1, 0), 50.0, W, H, 0.1, 100.0)
    ctx = gs.Context(0)
    scene = gs.Scene(ctx, sc["pos4"], sc["sr4"], gs.scenes.grouped_sh(sc["sh"]), 3)
    f = lambda *s: torch.zeros(s, dtype=torch.float32, device="cuda")  # noqa: E731
    xy, z, ell, conic, color = f(n, 2), f(n), f(n, 4), f(n, 4), f(n, 4)
    img = torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda")
    gs.probe_frame(ctx, scene, [cam], rc, [img], xy, z, ell, conic, color)
    h = lambda t: t.cpu().numpy()  # noqa: E731
    keys, vals = O.build(h(xy), h(ell), h(z), cam, rc)
    tiles = gs.num_tiles(W, H, rc)
    keys, vals = O.sort(keys, vals, gs.key_bits(tiles))
    ref = O.raster(cam, rc, O.ranges(keys, tiles), vals, h(xy), h(conic), h(color))
    scene.close()
    ctx.close()
    # the image bar of this mode: the culled contributions are each below 2^-18
    # and the stop below t_min, together within two 8-bit steps
    diff = np.abs(h(img).astype(int) - ref.astype(int))
    assert diff.max() <= 2, diff.max()
