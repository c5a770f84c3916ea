"""The tile lists of bucket frames whose splats cover one tile up to the whole
screen, against the oracle's build of the frame's own projected floats: every
(tile, depth, Gaussian) entry, in a context's first frame (whose lists are too
short at first) and in the next one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(gs, n, mu, sigma, seed):
    sc = gs.scenes.uniform_scene(n, seed=seed, log_scale_mu=mu, log_scale_sigma=sigma)
    sc["sr4"][::7, 1] *= 1e-3  # needles: many candidates, few overlaps
    sc["sr4"][3::11, :3] = 1e-7  # below a pixel: only the tile of the centre
    return sc


# tiles of 16x16 on 720x500: rectangles around 32 candidates (a warp's own walk
# against the large splats' kernel) and 1024 (one unit of that kernel or two)
@pytest.mark.parametrize("n,mu,sigma", [(1, -3.0, 0.1), (37, -1.6, 0.6), (3000, -3.6, 0.4), (3000, -2.6, 0.3),
                                        (20_000, -4.5, 1.2), (700, -0.9, 0.5)])
@pytest.mark.parametrize("mode", ["tmin", "ref"])
@pytest.mark.parametrize("views", [1, 3])
def test_tile_lists(gs, O, n, mu, sigma, mode, views):
    import torch
    sc = _scene(gs, n, mu, sigma, n + int(-mu * 10))
    rc = gs.RenderConfig() if mode == "tmin" else gs.RenderConfig.reference()
    sizes = [(720, 500), (333, 181), (64, 17)][:views]
    cams = [gs.look_at((0.1 * k, 0.2, 2.2 - 0.5 * k), (0, 0, 0), (0, 1, 0), 60.0, w, h, 0.1, 100.0)
            for k, (w, h) in enumerate(sizes)]
    ctx = gs.Context(0)
    scene = gs.Scene(ctx, sc["pos4"], sc["sr4"], gs.scenes.grouped_sh(sc["sh"]), 3)
    f = lambda *s: torch.zeros(s, dtype=torch.float32, device="cuda")  # noqa: E731
    xy, z, ell, conic, color = f(views * n, 2), f(views * n), f(views * n, 4), f(views * n, 4), f(views * n, 4)
    outs = [torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda") for w, h in sizes]
    for _ in range(2):
        gs.probe_frame(ctx, scene, cams, rc, outs, xy, z, ell, conic, color)
        t = gs.probe_tile_lists(ctx)
        got_tile = np.repeat(np.arange(len(t["ranges"])), t["ranges"][:, 1] - t["ranges"][:, 0])
        got_gi = t["slot_index"][(t["keys"] & np.uint64(0xFFFFFFFF)).astype(np.int64)]
        got = np.stack([got_tile, (t["keys"] >> np.uint64(32)).astype(np.int64), got_gi])
        want, offset, reached = [], 0, np.zeros(views * n, bool)
        for k, cam in enumerate(cams):
            part = slice(k * n, (k + 1) * n)
            keys, vals = O.build(xy[part].cpu().numpy(), ell[part].cpu().numpy(), z[part].cpu().numpy(), cam, rc)
            want.append(np.stack([(keys >> np.uint64(32)).astype(np.int64) + offset,
                                  (keys & np.uint64(0xFFFFFFFF)).astype(np.int64), vals.astype(np.int64) + k * n]))
            reached[k * n + vals] = True
            offset += gs.num_tiles(*sizes[k], rc)
        want = np.concatenate(want, 1)
        order = lambda a: a[:, np.lexsort(a[::-1])]  # noqa: E731
        assert np.array_equal(order(got), order(want))
        # the colours are those of the Gaussians that reach a tile
        assert np.array_equal((color.cpu().numpy() != 0).any(1), reached)
    scene.close()
    ctx.close()


# Needles of a minor extent far below a pixel: many candidates are too close to
# call and settled in the second walk, in early steps of a warp's walk and, at
# the longer extents, in steps from 31 on.
@pytest.mark.parametrize("n,length", [(1, 400.0), (33, 30.0), (33, 900.0), (5000, 12.0), (2000, 250.0)])
@pytest.mark.parametrize("width", [1e-3, 0.2])
def test_stage_build_of_needles(gs, O, n, length, width):
    import torch
    rng = np.random.default_rng(n + int(length))
    w, h = 720, 500
    cam = gs.look_at((0, 0, 2), (0, 0, 0), (0, 1, 0), 60.0, w, h, 0.1, 100.0)
    rc = gs.RenderConfig.reference()
    xy = (rng.random((n, 2)) * (w, h)).astype(np.float32)
    a = rng.random(n) * np.pi
    ell = np.stack([np.cos(a), np.sin(a), length * (0.5 + rng.random(n)), np.full(n, width)], 1).astype(np.float32)
    z = rng.random(n).astype(np.float32)
    keys, vals = O.build(xy, ell, z, cam, rc)
    ctx = gs.Context(0)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    cap = max(len(keys), 1)
    dk, dv = torch.zeros(cap, dtype=torch.int64, device="cuda"), torch.zeros(cap, dtype=torch.int32, device="cuda")
    K = gs.stage_build(ctx, n, dev(xy), dev(z), dev(ell), cam, rc, dk, dv, cap)
    assert K == len(keys)
    assert np.array_equal(dk.cpu().numpy()[:K].view(np.uint64), keys) and np.array_equal(dv.cpu().numpy()[:K], vals)
    ctx.close()
