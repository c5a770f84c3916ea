"""How often a bucket frame is drawn twice because its lists were too short:
not at all on a context's first frame whose keys fit the first key list, and
with a camera that moves in no more often than the key list alone needs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIRST_KEYS = (1 << 20) + (1 << 18)  # a context's first key list, scenes of up to 2^20 items


def _scene(gs, ctx, kind, n, seed):
    if kind == "uniform":
        sc = gs.scenes.uniform_scene(n, seed=seed, log_scale_mu=-4.0, log_scale_sigma=0.5)
    else:
        sc = gs.scenes.cluster_scene(n, 64, 5.0, seed=seed)
    return gs.Scene(ctx, sc["pos4"], sc["sr4"], gs.scenes.grouped_sh(sc["sh"]), 3)


@pytest.mark.parametrize("kind,n,size,eye,fovy", [
    ("uniform", 100_000, (800, 800), (1.2, 0.9, 2.6), 60.0),  # 0.8M keys
    ("clusters", 600_000, (1600, 900), (5.0, 3.0, 8.1), 50.0),  # 1M keys
    ("uniform", 4096, (320, 240), (0.2, 0.1, 3.0), 60.0),
])
@pytest.mark.parametrize("mode", ["tmin", "ref"])
def test_first_frame_is_drawn_once(gs, kind, n, size, eye, fovy, mode):
    import torch
    W, H = size
    ctx = gs.Context(0)
    scene = _scene(gs, ctx, kind, n, 7)
    rc = gs.RenderConfig() if mode == "tmin" else gs.RenderConfig.reference()
    cam = gs.look_at(eye, (0, 0, 0), (0, 1, 0), fovy, W, H, 0.1, 100.0)
    st = gs.render(ctx, scene, cam, rc, torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda"))
    scene.close()
    ctx.close()
    assert 0 < st["num_keys"] <= FIRST_KEYS, st["num_keys"]
    assert st["attempts"] == 1


@pytest.mark.parametrize("kind,n,far,near,fovy", [("uniform", 200_000, 8.0, 1.5, 60.0),
                                                  ("clusters", 900_000, 30.0, 4.0, 50.0)])
def test_moving_in_redoes_what_the_keys_need(gs, kind, n, far, near, fovy):
    import torch
    W, H = 1280, 720
    ctx = gs.Context(0)
    scene = _scene(gs, ctx, kind, n, 9)
    out = torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda")
    redone, needed, capacity = 0, 0, FIRST_KEYS
    for d in np.geomspace(far, near, 60):
        cam = gs.look_at((0.3 * d, 0.2 * d, 0.93 * d), (0, 0, 0), (0, 1, 0), fovy, W, H, 0.1, 100.0)
        st = gs.render(ctx, scene, cam, gs.RenderConfig(), out)
        redone += st["attempts"] - 1
        if st["num_keys"] > capacity:  # a quarter more than needed, and the allocation's quarter
            needed += 1
            capacity = st["num_keys"] * 5 // 4 * 5 // 4
    scene.close()
    ctx.close()
    assert needed >= 1
    assert redone <= needed, (redone, needed)
