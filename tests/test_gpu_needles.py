"""Needles: splats whose overlap with many of their candidate tiles is too
close to call for the cheap test and is settled in a second walk, through the
stage build (whole lists, in order) and through bucket frames (entries of each
tile), against the oracle's build."""
import numpy as np
import pytest

from test_overlap_margin import _centre, _decide

pytestmark = pytest.mark.gpu

W, H = 720, 500  # 45 x 32 tiles


def _needles(n, length, seed):
    """Centres on the screen, extents of about `length` pixels by a thousandth
    of a pixel to two: from some 0.07 pixels down the test's margin leaves every
    candidate open.  A third lie along tile borders, to within a few ulps."""
    rng = np.random.default_rng(seed)
    px = np.array([2.0 / W, 2.0 / H])
    xy = rng.uniform(-0.98, 0.98, (n, 2))
    angle = rng.uniform(0, np.pi, n)
    ex = length * (0.5 + rng.random(n)) * px[0]
    ey = np.exp(rng.uniform(np.log(1e-3), np.log(2.0), n)) * px[1]
    ey[0] = 1e-3 * px[1]
    k = np.arange(n) % 3 == 2
    border = rng.integers(1, 31, n) * (16 * 2.0 / H) - 1.0
    angle[k] = 0.0
    xy[k, 1] = (border + rng.choice([-1.0, 0.0, 1.0], n) * ey + rng.integers(-3, 4, n) * 6e-8)[k]
    ell = np.stack([np.cos(angle), np.sin(angle), ex, ey], 1)
    return xy.astype(np.float32), ell.astype(np.float32), rng.random(n).astype(np.float32)


def _undecided(xy, ell, most):
    """Candidates that the cheap test leaves open, of the splats with at most
    `most` candidates (tests/test_overlap_margin.py restates the test)."""
    tc = np.float32([16 * 2.0 / W, 16 * 2.0 / H])
    cs, sn, ex, ey = np.abs(ell.T)
    half = np.stack([cs * ex + sn * ey, sn * ex + cs * ey], 1)
    lo = np.maximum(np.floor((xy - half + 1) / tc), 0).astype(int)
    hi = np.minimum(np.ceil((xy + half + 1) / tc), [45, 32]).astype(int)
    cand = np.prod(np.maximum(hi - lo, 0), 1)
    open_, f = 0, np.float32
    for i in np.flatnonzero((cand > 0) & (cand <= most)):
        gx, gy = [g.ravel() for g in np.meshgrid(np.arange(lo[i, 0], hi[i, 0]), np.arange(lo[i, 1], hi[i, 1]))]
        x0, y0 = (gx.astype(f) * tc[0] - f(1)).astype(f), (gy.astype(f) * tc[1] - f(1)).astype(f)
        r = (x0, y0, (x0 + tc[0]).astype(f), (y0 + tc[1]).astype(f))
        e = [np.full(len(gx), v, f) for v in (xy[i, 0], xy[i, 1], *ell[i])]
        open_ += int(np.count_nonzero((_decide(e, r, 0) < 0) & ~_centre(e, r)))
    return open_, cand


# up to 32 candidates a splat; more; and walks of a warp of thousands, 45 x 32 tiles each
@pytest.mark.parametrize("n,length", [(1, 300.0), (33, 30.0), (33, 700.0), (5000, 12.0), (2000, 250.0)])
def test_stage_build(gs, O, n, length):
    import torch
    xy, ell, z = _needles(n, length, n + int(length))
    cam = gs.look_at((0, 0, 2), (0, 0, 0), (0, 1, 0), 60.0, W, H, 0.1, 100.0)
    rc = gs.RenderConfig.reference()
    keys, vals = O.build(xy, ell, z, cam, rc)
    open_, cand = _undecided(xy[:200], ell[:200], 1 << 20)
    assert len(keys) >= 2 * n and len(np.unique(vals)) >= 0.9 * n and open_ >= (n + 3) // 4 or open_ >= 50
    if length > 100 and n > 1:  # late steps of a warp's walk
        assert cand[:32].sum() > 32 * 32
    ctx = gs.Context(0)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    cap = len(keys)
    dk, dv = torch.zeros(cap, dtype=torch.int64, device="cuda"), torch.zeros(cap, dtype=torch.int32, device="cuda")
    K = gs.stage_build(ctx, n, dev(xy), dev(z), dev(ell), cam, rc, dk, dv, cap)
    ctx.close()
    assert K == len(keys)
    assert np.array_equal(dk.cpu().numpy().view(np.uint64), keys) and np.array_equal(dv.cpu().numpy(), vals)


@pytest.mark.parametrize("n,scale", [(40_000, 0.03), (20_000, 0.1)])
@pytest.mark.parametrize("mode", ["tmin", "ref"])
def test_bucket_frame(gs, O, n, scale, mode):
    import torch
    sc = gs.scenes.uniform_scene(n, seed=n)
    sc["sr4"][:, 0] = scale
    sc["sr4"][:, 1:3] = 1e-4
    rc = gs.RenderConfig() if mode == "tmin" else gs.RenderConfig.reference()
    cam = gs.look_at((0.1, 0.2, 2.4), (0, 0, 0), (0, 1, 0), 60.0, W, H, 0.1, 100.0)
    ctx = gs.Context(0)
    scene = gs.Scene(ctx, sc["pos4"], sc["sr4"], gs.scenes.grouped_sh(sc["sh"]), 3)
    f = lambda *s: torch.zeros(s, dtype=torch.float32, device="cuda")  # noqa: E731
    xy, z, ell, conic = f(n, 2), f(n), f(n, 4), f(n, 4)
    out = torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda")
    gs.probe_frame(ctx, scene, [cam], rc, [out], xy, z, ell, conic, f(n, 4))
    t = gs.probe_tile_lists(ctx)
    scene.close()
    ctx.close()
    h = lambda x: x.cpu().numpy()  # noqa: E731
    open_, cand = _undecided(h(xy), h(ell), 32)
    assert open_ >= 20 and np.count_nonzero((cand > 1) & (cand <= 32)) >= n // 4, open_
    keys, vals = O.build(h(xy), h(ell), h(z), cam, rc)
    tile = np.repeat(np.arange(len(t["ranges"])), t["ranges"][:, 1] - t["ranges"][:, 0])
    depth = (t["keys"] >> np.uint64(32)).astype(np.uint64)
    got = np.stack([tile.astype(np.uint64) << np.uint64(32) | depth,
                    t["slot_index"][(t["keys"] & np.uint64(0xFFFFFFFF)).astype(np.int64)].astype(np.uint64)])
    want = np.stack([keys, vals.astype(np.uint64)])
    order = lambda a: a[:, np.lexsort(a[::-1])]  # noqa: E731
    assert np.array_equal(order(got), order(want))
