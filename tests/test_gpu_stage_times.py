"""The stage times of a frame: every time is there, whatever the raster's
launch (one CTA per tile, persistent CTAs, several launches of a host-output
frame), and each is this frame's own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(st):
    assert st["raster_ms"] > 0
    assert st["total_ms"] >= st["raster_ms"] + st["project_ms"]
    parts = st["project_ms"] + st["build_tile_ms"] + st["sort_ms"] + st["raster_ms"]
    # the stages follow one another: the total is their sum (to the clock's step)
    assert abs(st["total_ms"] - parts) < 0.01, st


# 3600 and 32400 tiles of 16x16: more tiles than persistent CTAs
@pytest.mark.parametrize("size", [(64, 48), (1280, 720), (3840, 2160)])
@pytest.mark.parametrize("tile", [(16, 16), (16, 8), (8, 8)])
@pytest.mark.parametrize("persistent", [0, 1])
def test_stage_times(gs, size, tile, persistent):
    import torch
    W, H = size
    sc = gs.scenes.uniform_scene(20_000, seed=5)
    ctx = gs.Context(0)
    scene = gs.Scene(ctx, sc["pos4"], sc["sr4"], gs.scenes.grouped_sh(sc["sh"]), 3)
    rc = gs.RenderConfig(tile_w=tile[0], tile_h=tile[1], raster_persistent=persistent)
    cam = gs.look_at((0.1, 0.2, 2.5), (0, 0, 0), (0, 1, 0), 60.0, W, H, 0.1, 100.0)
    out = torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda")
    for _ in range(3):  # plain, captured, replayed
        _check(gs.render(ctx, scene, cam, rc, out))
    host = np.zeros((H, W, 4), np.uint8)
    for _ in range(3):  # the larger images in several raster launches
        _, st = gs.render_host(ctx, scene, cam, rc, host)
        _check(st)
    scene.close()
    ctx.close()


@pytest.mark.parametrize("mode", ["tmin", "ref"])
def test_raster_time_holds_the_longest_tile(gs, mode):
    """A tile of 40000 nearly transparent splats among 32400 empty ones: it is
    drawn first and ends last, long after the others.  The same tile alone on
    a small image says how long it takes."""
    import torch
    n = 40_000
    rng = np.random.default_rng(8)
    pos4 = np.empty((n, 4), np.float32)
    pos4[:, 0], pos4[:, 1] = 0.012, 0.009  # off the corner of four tiles
    pos4[:, 2] = rng.normal(0, 0.05, n)
    pos4[:, 3] = 1e-4  # T stays above exp(-4): no tile stops early
    sr4 = gs.scenes.uniform_scene(n, seed=1)["sr4"]
    sr4[:, :3] = 1e-3
    color4 = np.concatenate([rng.random((n, 3)), pos4[:, 3:]], 1).astype(np.float32)
    rc = gs.RenderConfig() if mode == "tmin" else gs.RenderConfig.reference()
    ctx = gs.Context(0)
    scene = gs.Scene(ctx, pos4, sr4, None, 0, color4)
    times = []
    for W, H in ((256, 144), (3840, 2160)):
        cam = gs.look_at((0, 0, 2.5), (0, 0, 0), (0, 1, 0), 60.0, W, H, 0.1, 100.0)
        out = torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda")
        st = [gs.render(ctx, scene, cam, rc, out) for _ in range(4)]
        times.append(min(s["raster_ms"] for s in st[1:]))
    scene.close()
    ctx.close()
    # the lanes of a large launch draw twice the pixels each: no faster
    assert times[1] > 0.8 * times[0], times
