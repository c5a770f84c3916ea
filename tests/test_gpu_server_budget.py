"""A burst of requests whose scene has tens of tile-list keys per Gaussian is
cut into batches whose buffers stay within the server's budget."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_burst_stays_within_the_budget(gs):
    import torch
    W, H = 640, 480
    sc = gs.scenes.uniform_scene(60_000, seed=3, log_scale_mu=-2.0, log_scale_sigma=0.3)
    sh = gs.scenes.grouped_sh(sc["sh"])
    cams = [gs.look_at((0.1 * k, 0.2, 3.0), (0, 0, 0), (0, 1, 0), 60.0, W, H, 0.1, 100.0) for k in range(16)]
    ctx = gs.Context(0)  # the library is loaded and has run
    scene = gs.Scene(ctx, sc["pos4"], sc["sr4"], sh, 3)
    want, st = gs.render_host(ctx, scene, cams[-1], gs.RenderConfig())
    assert st["num_keys"] > 20 * 60_000, st["num_keys"]
    scene.close()
    ctx.close()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    budget = 1 << 30
    srv = gs.Server(0, budget_bytes=budget, max_batch_views=16, num_workers=1, batch_target_ms=0.0)
    sid = srv.add_scene(sc["pos4"], sc["sr4"], sh, 3)
    outs = [np.zeros((H, W, 4), np.uint8) for _ in cams]
    for _ in range(12):  # the server learns the scene's keys per Gaussian
        srv.wait(srv.submit(sid, cams[0], outs[0]))
    srv.pause()
    ids = [srv.submit(sid, c, o) for c, o in zip(cams, outs)]
    srv.pause(False)
    for i in ids:
        srv.wait(i)
    held = free0 - torch.cuda.mem_get_info()[0]
    assert srv.stats()["max_batch"] >= 2
    srv.close()
    assert np.array_equal(outs[-1], want)
    # 32 MB for the granularity of the device's allocations
    assert held <= budget + (32 << 20), held
