"""The work a program has this framework do, as cases that can be timed:
single views, batches of views, host-memory output, the stage API and the
render server, from a few thousand Gaussians to ten million.

A case is a dict of plain values; `prepare` builds the scene, cameras,
context and outputs it needs from a seed, `run` does one pass through the
public entry points and returns everything it computed.  Scenes come from
the generators of the benchmark configurations (uniform cube or anisotropic
clusters, log-normal scales, random quaternions, opacity = sigmoid(N(0, 1.5)),
SH DC ~ N(0, 0.5), rest ~ N(0, 0.05)), drawn on the GPU so that they are
quick to make.
"""
import importlib
import math

import numpy as np
import torch

gs = importlib.import_module("3dgaussianrenderer_b200")

MIXED = ((1280, 720), (1600, 900), (1920, 1080))
SERVED = ((1280, 720), (1920, 1080), (2560, 1440))


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def _case(name, kind, n, w, h, views=1, gen="clusters", clusters=64, extent=5.0, mu=-5.0, sigma=0.7, degree=3,
          dist=10.0, fovy=50.0, mixed=False, mode="tmin", tile_w=16, tile_h=16, chunk=0, vpb=0, ordering="buckets",
          keep_order=False):
    c = dict(name=name, kind=kind, n=n, w=w, h=h, views=views, gen=gen, clusters=clusters, extent=extent, mu=mu,
             sigma=sigma, degree=degree, dist=dist, fovy=fovy, mixed=mixed, mode=mode, tile_w=tile_w, tile_h=tile_h,
             chunk=chunk, vpb=vpb, ordering=ordering, keep_order=keep_order)
    if name is None:
        del c["name"]
    return c


def listed():
    cube = dict(gen="uniform", clusters=0, extent=1.0, mu=-4.0, sigma=0.5, dist=3.0, fovy=60.0)
    big = dict(clusters=256, extent=10.0, dist=15.0)
    return [
        # a preview or a unit test: a few thousand splats, where launches and the host path are the cost
        _case("view_4k_320x240", "view", 4096, 320, 240, **cube),
        # the smallest benchmark scene, one view on the screen of a small application
        _case("view_100k_800x800", "view", 100_000, 800, 800, **cube),
        # an ordinary captured object at full HD, one view
        _case("view_1m_1920x1080", "view", 1_000_000, 1920, 1080),
        # the drop-in frame of the reference renderer: its image size, its SH degree and termination
        _case("ref_view_3m_1024x1024", "view", 3_000_000, 1024, 1024, mode="ref", **big),
        # a viewer without a GPU display: colour-only model, odd image size, image back in host memory
        _case("ref_host_300k_deg0_1001x701", "view_host", 300_000, 1001, 701, degree=0, mode="ref"),
        # dataset rendering, the headline workload: 64 views of a large scene in one frame, with the knobs its
        # autotuner picks (32 views per block, 64-entry raster chunks)
        _case("batch64_3m_mixed", "batch", 3_000_000, 1920, 1080, views=64, mixed=True, chunk=64, vpb=32, **big),
        # a batch of novel views written to host memory (video, evaluation), default knobs
        _case("batch24_host_1m_mixed", "batch_host", 1_000_000, 1920, 1080, views=24, mixed=True),
        # several small odd-sized views per frame in the reference's termination, SH degree 2
        _case("ref_batch5_500k_sh2_637x479", "batch", 500_000, 637, 479, views=5, degree=2, mode="ref"),
        # the reference's own list order (keys in Gaussian order, one radix sort), scene in caller order
        _case("onesweep_batch8_1m_1280x720", "batch", 1_000_000, 1280, 720, views=8, ordering="onesweep",
              keep_order=True),
        # ten million large, heavily overlapping splats at 4K: the longest tile lists
        _case("view_10m_large_3840x2160", "view", 10_000_000, 3840, 2160, clusters=256, extent=10.0, mu=-2.5,
              sigma=0.8, dist=15.0),
        # an application with its own frame loop on the stage API, all six stages in the reference's layouts
        _case("stages_1m_1024x1024", "stages", 1_000_000, 1024, 1024, mode="ref"),
        # a burst of 24 requests to the render server over four resident scenes (n is the largest)
        _case("serve_24_requests", "serve", 2_000_000, 2560, 1440, views=24, dist=12.0, clusters=256, extent=10.0),
    ]


def draw(rng):
    """One more case: sizes over the ranges above (log-uniform), every kind and option."""
    def logu(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["view", "view", "view_host", "batch", "batch", "batch_host", "stages", "serve"])
    mode = "ref" if kind == "stages" else rng.choice(["tmin", "tmin", "ref"])
    if kind == "stages":
        n, w = logu(2000, 1_000_000), logu(240, 1280)
    elif kind == "serve":
        n, w = logu(20_000, 2_000_000), 2560
    elif kind in ("batch", "batch_host"):
        n, w = logu(4000, 2_000_000), logu(200, 1600)
    else:
        n, w = logu(2000, 3_000_000), logu(200, 3000)
    h = max(16, int(w * rng.uniform(0.5, 1.0)))
    views = {"view": 1, "view_host": 1, "stages": 1, "serve": rng.randint(6, 20), "batch": rng.randint(2, 32),
             "batch_host": rng.randint(2, 32)}[kind]
    degree = rng.choice([1, 2, 3, 3, 3] if kind == "stages" else [0, 1, 2, 3, 3, 3])
    # other tile shapes, raster chunks and views per block are the autotuner's choices for T_min batches
    tile_w, tile_h = rng.choice([(16, 16), (16, 16), (16, 16), (16, 8), (8, 8)]) if mode == "tmin" else (16, 16)
    ordering = "onesweep" if kind in ("view", "batch") and rng.random() < 0.15 else "buckets"
    chunk, vpb = (rng.choice([0, 32, 64]), rng.choice([0, 8, 32])) if kind.startswith("batch") else (0, 0)
    if rng.random() < 0.35:
        scene = dict(gen="uniform", clusters=0, extent=1.0, mu=round(rng.uniform(-4.8, -3.8), 2), sigma=0.5,
                     dist=round(rng.uniform(2.5, 4.0), 2), fovy=60.0)
    else:
        extent = round(rng.uniform(4.0, 10.0), 1)
        scene = dict(clusters=rng.choice([64, 128, 256]), extent=extent, mu=round(rng.uniform(-5.3, -4.3), 2),
                     sigma=0.7, dist=round(extent * rng.uniform(1.3, 2.2), 1))
    return _case(None, kind, n, w, h, views=views, degree=degree, mode=mode, tile_w=tile_w, tile_h=tile_h,
                 chunk=chunk, vpb=vpb, ordering=ordering, keep_order=ordering == "onesweep",
                 mixed=kind.startswith("batch") and rng.random() < 0.3, **scene)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _sizes(case):
    """(width, height) of every view."""
    if case["kind"] == "serve":
        return [SERVED[i % 3] for i in range(case["views"])]
    if case["mixed"]:
        return [MIXED[i % 3] for i in range(case["views"])]
    return [(case["w"], case["h"])] * case["views"]


def _scene(case, n, seed):
    """A scene's arrays on the GPU, in the framework's layouts."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    def uniform(lo, hi, *shape):
        return torch.rand(*shape, generator=g, device="cuda") * (hi - lo) + lo

    e = case["extent"]
    if case["gen"] == "uniform":
        means = uniform(-e, e, n, 3)
    else:
        k = case["clusters"]
        centres, var = uniform(-e, e, k, 3), uniform(0.05, 1.0, k, 3)
        which = torch.randint(0, k, (n,), generator=g, device="cuda")
        means = centres[which] + normal(n, 3) * var[which].sqrt()
    opacity = torch.sigmoid(normal(n) * 1.5)
    scale = torch.exp(normal(n, 3) * case["sigma"] + case["mu"])
    q = normal(n, 4)
    q = q / q.norm(dim=1, keepdim=True)  # (x, y, z, w), one byte a component
    b = (((q + 1) * 0.5).clamp(0, 1) * 255).to(torch.int64)
    bits = (b[:, 0] << 24) | (b[:, 1] << 16) | (b[:, 2] << 8) | b[:, 3]
    bits = torch.where(bits >= 1 << 31, bits - (1 << 32), bits).to(torch.int32)
    pos4 = torch.cat([means, opacity[:, None]], 1).contiguous()
    sr4 = torch.cat([scale, bits.view(torch.float32)[:, None]], 1).contiguous()
    d = case["degree"]
    if d == 0:
        color4 = torch.cat([normal(n, 3) * 0.5 * 0.28209479 + 0.5, opacity[:, None]], 1).contiguous()
        return dict(pos4=pos4, sr4=sr4, color4=color4, sh=None)
    c = 3 * (d + 1) ** 2
    groups = (n + 255) // 256
    sh = normal(groups, c, 256)  # grouped: [group][coefficient][256], zero past the last Gaussian
    sh[:, :3] *= 0.5
    sh[:, 3:] *= 0.05
    if n % 256:
        sh[-1, :, n % 256:] = 0
    return dict(pos4=pos4, sr4=sr4, color4=None, sh=sh.reshape(-1))


def _host(x):
    return None if x is None else x.cpu().numpy()


def _cameras(case, seed):
    rng = np.random.default_rng(seed)
    sizes = _sizes(case)
    if case["kind"].startswith("batch"):
        eyes = gs.scenes.orbit_ring(len(sizes), case["dist"], seed)
    else:
        eyes = [gs.scenes.sphere_pose(rng, case["dist"]) for _ in sizes]
    return [gs.look_at(e, (0, 0, 0), (0, 1, 0), case["fovy"], w, h, 0.1, 100.0) for e, (w, h) in zip(eyes, sizes)]


def _config(case):
    c = gs.RenderConfig.reference() if case["mode"] == "ref" else gs.RenderConfig()
    c.tile_w, c.tile_h = case["tile_w"], case["tile_h"]
    c.raster_chunk, c.views_per_block = case["chunk"], case["vpb"]
    c.ordering = gs.GS_ORDER_ONESWEEP if case["ordering"] == "onesweep" else gs.GS_ORDER_BUCKETS
    return c


def _pinned(nbytes):
    return torch.empty(nbytes, dtype=torch.uint8).pin_memory().numpy()


def _list_capacity(case):
    """Tile-list entries to allocate for a view: 2.5 times the mean number of
    16-pixel tiles a splat's 3-sigma square spans at the scene's centre."""
    f = 0.5 * case["h"] / math.tan(math.radians(case["fovy"]) / 2)
    k, mu, v = 6 * f / case["dist"] / 16, case["mu"], case["sigma"] ** 2
    spans = 1 + 2 * k * math.exp(mu + v / 2) + k * k * math.exp(2 * mu + 2 * v)
    return int(2.5 * spans * case["n"]) + (1 << 16)


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    cams, sizes = _cameras(case, seed), _sizes(case)
    s = dict(kind=kind, cams=cams, cfg=_config(case))
    if kind == "serve":
        cfg = _config(case)
        cfg.graph = 0  # the server's default: its batches rarely repeat
        s["server"] = gs.Server(0, budget_bytes=60 << 30, max_batch_views=16, num_workers=2, cfg=cfg)
        ids = []
        for k, m in enumerate((n // 10, n // 4, n // 2, n)):
            sc = _scene(case, m, seed * 4 + k)
            ids.append(s["server"].add_scene(_host(sc["pos4"]), _host(sc["sr4"]), _host(sc["sh"]), case["degree"],
                                             _host(sc["color4"])))
        s["ids"] = [ids[int(k)] for k in np.random.default_rng(seed + 1).integers(0, 4, len(cams))]
        s["outs"] = [_pinned(4 * w * h).reshape(h, w, 4) for w, h in sizes]
        return s
    sc = _scene(case, n, seed)
    s["ctx"] = gs.Context(0)
    if kind == "stages":
        # a frame loop of its own keeps the model, every stage's buffer and lists sized with room
        dev = dict(device="cuda")
        w, h = sizes[0]
        cap = _list_capacity(case)
        tiles = gs.num_tiles(w, h, s["cfg"])
        s.update(n=n, pos=sc["pos4"], sr=sc["sr4"], sh=sc["sh"], sh_count=3 * (case["degree"] + 1) ** 2,
                 degree=min(case["degree"], 2), cap=cap, tiles=tiles, bits=gs.key_bits(tiles),
                 color=torch.zeros(n, 4, **dev), xy=torch.zeros(n, 2, **dev), z=torch.zeros(n, **dev),
                 ell=torch.zeros(n, 4, **dev), conic=torch.zeros(n, 4, **dev),
                 keys=[torch.zeros(cap, dtype=torch.int64, **dev) for _ in range(2)],
                 vals=[torch.zeros(cap, dtype=torch.int32, **dev) for _ in range(2)],
                 ranges=torch.zeros(tiles, 2, dtype=torch.int32, **dev),
                 rgba=torch.zeros(h, w, 4, dtype=torch.uint8, **dev))
        return s
    s["scene"] = gs.Scene(s["ctx"], _host(sc["pos4"]), _host(sc["sr4"]), _host(sc["sh"]), case["degree"],
                          _host(sc["color4"]), keep_order=case["keep_order"])
    if kind.endswith("_host"):
        s["out"] = _pinned(sum(4 * w * h for w, h in sizes))
    else:
        s["outs"] = [torch.zeros(h, w, 4, dtype=torch.uint8, device="cuda") for w, h in sizes]
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _stages(s):
    n, cam = s["n"], s["cams"][0]
    gs.stage_sh(n, s["pos"], s["sh"], s["sh_count"], s["degree"], cam, s["color"])
    gs.stage_project(n, s["pos"], s["sr"], cam, s["xy"], s["z"], s["ell"], s["conic"])
    k = gs.stage_build(s["ctx"], n, s["xy"], s["z"], s["ell"], cam, s["cfg"], s["keys"][0], s["vals"][0], s["cap"])
    side = gs.stage_sort(s["ctx"], k, s["bits"], s["keys"][0], s["vals"][0], s["keys"][1], s["vals"][1])
    keys, vals = s["keys"][side], s["vals"][side]
    gs.stage_ranges(k, keys, s["tiles"], s["ranges"])
    s["rgba"].zero_()
    gs.stage_raster(cam, s["cfg"], s["ranges"], vals, s["xy"], s["conic"], s["color"], s["rgba"])
    # the lists come back at their capacity (zero past the last key): their length is the scene's
    return dict(color=s["color"], xy=s["xy"], z=s["z"], ell=s["ell"], conic=s["conic"], keys=keys, values=vals,
                ranges=s["ranges"], rgba=s["rgba"], num_keys=k)


def run(state):
    s = state
    kind = s["kind"]
    if kind == "view":
        gs.render(s["ctx"], s["scene"], s["cams"][0], s["cfg"], s["outs"][0])
        return s["outs"][0]
    if kind == "batch":
        gs.render_batch(s["ctx"], s["scene"], s["cams"], s["cfg"], s["outs"])
        return s["outs"]
    if kind == "view_host":
        gs.render_host(s["ctx"], s["scene"], s["cams"][0], s["cfg"], s["out"])
        return s["out"]
    if kind == "batch_host":
        gs.render_batch_host(s["ctx"], s["scene"], s["cams"], s["cfg"], s["out"])
        return s["out"]
    if kind == "stages":
        return _stages(s)
    server = s["server"]
    ids = [server.submit(i, cam, out) for i, cam, out in zip(s["ids"], s["cams"], s["outs"])]
    for i in ids:
        server.wait(i)
    return s["outs"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    """Bytes: every Gaussian's attributes read once, every pixel written once
    (the stage API also writes its per-Gaussian buffers).  Flops: projection
    (250) and SH per view and Gaussian, and the blend (20 per evaluation) of
    the pixels inside each splat's 3-sigma ellipse, at most the 25 or so
    evaluations after which a pixel of mean opacity 1/2 is opaque."""
    n, d = case["n"], case["degree"]
    per = 32 + (16 if d == 0 else 12 * (d + 1) ** 2)
    sizes = _sizes(case)
    px = sum(w * h for w, h in sizes)
    total = n
    if case["kind"] == "serve":
        total = n // 10 + n // 4 + n // 2 + n
    gauss = n * len(sizes) if case["kind"] != "serve" else total * len(sizes) / 4
    nbytes = total * per + 4 * px
    if case["kind"] == "stages":
        nbytes += n * (16 + 8 + 4 + 16 + 16)
    s2 = math.exp(2 * case["mu"] + case["sigma"] ** 2)  # mean product of two of a splat's scales
    evals = 0.0
    for w, h in sizes:
        f = 0.5 * h / math.tan(math.radians(case["fovy"]) / 2)
        foot = 9 * math.pi * (s2 * f * f / case["dist"] ** 2 + 0.4)
        evals += min(gauss / len(sizes) * foot, 25.0 * w * h)
    sh = 0 if d == 0 else 6 * (d + 1) ** 2 + 30
    return {"bytes": float(nbytes), "flops": float(gauss * (250 + sh) + 20 * evals)}


# ---------------------------------------------------------------------------
# exact values of the stage API's floating-point outputs
# ---------------------------------------------------------------------------

_SH = [
    lambda x, y, z: torch.full_like(x, 0.282094792),
    lambda x, y, z: 0.488602512 * y,
    lambda x, y, z: 0.488602512 * z,
    lambda x, y, z: 0.488602512 * x,
    lambda x, y, z: 1.09254843 * x * y,
    lambda x, y, z: 1.09254843 * y * z,
    lambda x, y, z: -0.946174696 * x * x - 0.946174696 * y * y + 0.630783131,
    lambda x, y, z: 1.09254843 * x * z,
    lambda x, y, z: 0.546274215 * (x - y) * (x + y),
]


def _project64(pos, sr, cam):
    """Clip-space centre, ellipse and conic of every Gaussian in 64 bits."""
    c = cam.c
    t = lambda v, *shape: torch.tensor(list(v), dtype=torch.float64, device="cuda").reshape(*shape)  # noqa: E731
    view = t(c.view, 4, 4).T  # rows
    p = pos[:, :3].double()
    v = p @ view[:3, :3].T + view[:3, 3]
    cot, dsb = t(c.fov_cotangent, 2), t(c.depth_scale_bias, 2)
    rz = 1.0 / v[:, 2]
    xy = -cot * v[:, :2] * rz[:, None]
    z = dsb[0] * v[:, 2] + dsb[1]
    bits = sr[:, 3].contiguous().view(torch.int32).to(torch.int64)
    q = torch.stack([(bits >> k) & 255 for k in (24, 16, 8, 0)], 1).double() / 255 * 2 - 1
    x, y, zq, w = q.unbind(1)
    R = torch.stack([1 - 2 * (y * y + zq * zq), 2 * (x * y - w * zq), 2 * (x * zq + w * y),
                     2 * (x * y + w * zq), 1 - 2 * (x * x + zq * zq), 2 * (y * zq - w * x),
                     2 * (x * zq - w * y), 2 * (y * zq + w * x), 1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)
    rs = R * sr[:, None, :3].double()
    J = torch.zeros(len(p), 2, 3, dtype=torch.float64, device="cuda")
    J[:, 0, 0], J[:, 1, 1] = -cot[0] * rz, -cot[1] * rz
    J[:, 0, 2], J[:, 1, 2] = cot[0] * v[:, 0] * rz * rz, cot[1] * v[:, 1] * rz * rz
    m = J @ view[:3, :3] @ rs
    cov = m @ m.transpose(1, 2)
    c00 = cov[:, 0, 0] + (2.0 / c.width) ** 2 / 3.14159265359
    c11 = cov[:, 1, 1] + (2.0 / c.height) ** 2 / 3.14159265359
    c10 = cov[:, 0, 1]
    det, mid = c00 * c11 - c10 * c10, 0.5 * (c00 + c11)
    r = (mid * mid - det).clamp(min=1e-12).sqrt()
    l0, l1 = mid + r, (mid - r).clamp(min=0)
    e = torch.stack([c10, l0 - c00], 1)
    e = e / e.norm(dim=1, keepdim=True)
    inv = 1.0 / det.clamp(min=1e-12)
    seen = ((xy.abs() <= 1).all(1) & (z.abs() <= 1)).double()
    ell = torch.stack([e[:, 0], e[:, 1], 3 * l0.sqrt() * seen, 3 * l1.sqrt() * seen], 1)
    conic = torch.stack([c11 * inv, -c10 * inv, c00 * inv, torch.zeros_like(inv)], 1)
    out = lambda a: torch.where(seen > 0, a, torch.full_like(a, -128.0))  # noqa: E731
    return torch.stack([out(xy[:, 0]), out(xy[:, 1])], 1), out(z), ell, conic


def exact(case, seed):
    """The stage API's colours and projections in 64 bits; lists, ranges and
    images are whole numbers and bytes and have no value here."""
    if case["kind"] != "stages":
        return None
    sc = _scene(case, case["n"], seed)
    cam = _cameras(case, seed)[0]
    pos, n, d = sc["pos4"], case["n"], case["degree"]
    eye = torch.tensor(list(cam.c.position), dtype=torch.float64, device="cuda")
    dirs = eye - pos[:, :3].double()
    x, y, z = (dirs / dirs.norm(dim=1, keepdim=True)).unbind(1)
    c = 3 * (d + 1) ** 2
    sh = sc["sh"].reshape(-1, c, 256).permute(0, 2, 1).reshape(-1, c // 3, 3)[:n].double()
    rgb = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
    for k in range((min(d, 2) + 1) ** 2):
        rgb += _SH[k](x, y, z)[:, None] * sh[:, k]
    color = torch.cat([(rgb + 0.5).clamp(0, 1), pos[:, 3:].double()], 1)
    xy, zc, ell, conic = _project64(pos, sc["sr4"], cam)
    return dict(color=color, xy=xy, z=zc, ell=ell, conic=conic, keys=None, values=None, ranges=None, rgba=None,
                num_keys=None)
