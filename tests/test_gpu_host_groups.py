"""Host-output frames stream their images in groups of tile rows: the images
are those of the device-output frame, whatever the groups cut."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [{}, {"tile_w": 8, "tile_h": 8}, {"raster_persistent": 1}, {"termination": 0}])
# below one group; cut inside a view and inside the last one; more than the most
# groups; a width that leaves the rows unaligned
@pytest.mark.parametrize("sizes", [[(200, 100)], [(1001, 701), (64, 3001), (333, 17)], [(2001, 1403)] * 4, [(3, 1)] * 3])
def test_host_output_equals_device_output(gs, kw, sizes):
    import torch
    sc = gs.scenes.uniform_scene(3000, seed=4)
    ctx = gs.Context(0)
    scene = gs.Scene(ctx, sc["pos4"], sc["sr4"], gs.scenes.grouped_sh(sc["sh"]), 3)
    rc = gs.RenderConfig(**kw)
    cams = [gs.look_at((0.1 * k, 0.2, 2.5), (0, 0, 0), (0, 1, 0), 60.0, w, h, 0.1, 100.0)
            for k, (w, h) in enumerate(sizes)]
    outs = [torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda") for w, h in sizes]
    gs.render_batch(ctx, scene, cams, rc, outs)
    want = np.concatenate([o.cpu().numpy().reshape(-1) for o in outs])
    for _ in range(3):  # plain, captured, replayed
        got = np.full(want.size, 7, np.uint8)
        gs.render_batch_host(ctx, scene, cams, rc, got)
        assert np.array_equal(got, want)
    if len(sizes) == 1:
        got, _ = gs.render_host(ctx, scene, cams[0], rc)
        assert np.array_equal(got.reshape(-1), want)
    scene.close()
    ctx.close()
