"""The blend order of tiles of tens of thousands of entries, which are sorted
ahead of the raster in parts of 16384 keys or, beyond 65535 and with long runs
of close depths, by passes through global memory: depth first, caller index
among equal depths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _depths(kind, m, rng):
    """Distances from the camera; the depth key's top bit changes at 50.05."""
    if kind == "spread":
        return rng.uniform(1.0, 90.0, m)
    if kind == "edge":  # the first part ends with the 16384th key, at a bin's end
        return np.concatenate([rng.uniform(20.0, 45.0, 16384), rng.uniform(55.0, 80.0, m - 16384)])
    if kind == "runs":  # 40 keys of each depth
        return 10.0 + 0.05 * (np.arange(m) // 40)
    if kind == "long":  # one depth more often than a part holds keys
        return np.concatenate([np.full(16385, 33.0), rng.uniform(20.0, 45.0, m - 16385)])
    return np.full(m, 33.0)


@pytest.mark.parametrize("kind", ["spread", "edge", "runs", "long", "equal"])
@pytest.mark.parametrize("m", [16384, 16385, 20_000, 32_768, 40_000, 65_535, 65_536])
def test_order_of_a_large_tile(gs, kind, m):
    import torch
    if m < 16385 and kind == "long":
        pytest.skip("fewer keys than the run")
    rng = np.random.default_rng(m)
    dist = rng.permutation(_depths(kind, m, rng)).astype(np.float32)
    W = H = 64
    cam = gs.look_at((0, 0, 0), (0, 0, -1), (0, 1, 0), 60.0, W, H, 0.1, 100.0)
    # every centre at clip (0.25, 0.25), the middle of one 16x16 tile, far below a pixel wide
    pos4 = np.empty((m, 4), np.float32)
    pos4[:, 0] = pos4[:, 1] = 0.25 * np.tan(np.radians(30.0)) * dist
    pos4[:, 2] = -dist
    pos4[:, 3] = 0.5
    sr4 = gs.scenes.uniform_scene(m, seed=1)["sr4"]
    sr4[:, :3] = 1e-6
    ctx = gs.Context(0)
    scene = gs.Scene(ctx, pos4, sr4, None, 0, np.full((m, 4), 0.5, np.float32))
    f = lambda *s: torch.zeros(s, dtype=torch.float32, device="cuda")  # noqa: E731
    xy, z, ell, conic = f(m, 2), f(m), f(m, 4), f(m, 4)
    img = torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        gs.probe_frame(ctx, scene, [cam], gs.RenderConfig(), [img], xy, z, ell, conic, f(m, 4))
        t = gs.probe_tile_lists(ctx)
        counts = t["ranges"][:, 1] - t["ranges"][:, 0]
        assert counts.max() == m == counts.sum()
        got = t["slot_index"][t["order"]]
        zz = z.cpu().numpy()
        key = ((zz + np.float32(1)) * np.float32(0.5)).astype(np.float32) * np.float32(2.0 ** 32)
        assert np.array_equal(got, np.lexsort((np.arange(m), key)))
    scene.close()
    ctx.close()
