"""The work that programs using this framework have it do, as timed cases.

A case is a dict of plain values; ``kind`` says which calls it makes:

  frame   the breadth-first renderer's batches on device buffers: one camera
          batch (nearest hit), then one shadow batch (any hit) per light
          sample, for any of the three accelerators
  tile    the same for one task tile through the host-array calls that pbrt's
          batch integrators make: Intersect, HitGeometry, IntersectP
  bounce  a path bounce on device buffers: nearest hit with a validity mask,
          and the shadow rays that leave the same points
  render  a whole image through the device renderer (path or directlighting)
  set     many independent scenes answered by one call
  train   SGD steps of the learned traversal ordering on collected records
  ordered shadow rays walked in the learned order (inference and walk)

Scenes are seeded: a fractal height field with icospheres on it, displaced
icospheres in a box, or a sphere over a ground quad.  Camera rays come in
scanline order with the samples of a pixel side by side, shadow rays leave
the camera's hits, bounce rays leave them in cosine-weighted directions: the
order and coherence that a renderer's batches have.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

import pbg_import

pbg_import.load()
from pbrt_gb300 import _lib as L  # noqa: E402
from pbrt_gb300 import accel as A  # noqa: E402
from pbrt_gb300 import batch as B  # noqa: E402
from pbrt_gb300 import render as R  # noqa: E402
from pbrt_gb300 import scenes as S  # noqa: E402

NPARAM = 64 * 112 + 64 + 64 * 64 + 64 + 256 * 64 + 256
SPHERE_TRIS = 1280  # an icosphere at subdivision 3


def listed():
    return [
        # one pick or probe call of an interactive program: a few hundred rays, where latency is all
        dict(name="pick_500", kind="frame", accel="ray-bvh", scene="terrain", tris=20000, w=25, h=20, spp=1, lights=0),
        # the small brute-force image: sphere over a ground quad, 256 x 256 at pixel centres, one point light
        dict(name="naive_256", kind="frame", accel="naive", scene="sphere", tris=4034, w=256, h=256, spp=1, lights=1),
        # a preview tile of an odd size through the ray hierarchy
        dict(name="hier_preview", kind="frame", accel="rayhierarchy", scene="terrain", tris=12000, w=161, h=119, spp=1, lights=1),
        # the ray-hierarchy frame: 1024 x 1024 at 4 samples, terrain with 40 spheres, 4 area-light samples
        dict(name="hier_frame", kind="frame", accel="rayhierarchy", scene="terrain", tris=181250, w=1024, h=1024, spp=4, lights=4),
        # one task tile (MaxRaysPerCall rays) of pbrt's breadth-first renderer, host arrays in and out
        dict(name="tile_host", kind="tile", accel="ray-bvh", scene="terrain", tris=181250, w=640, h=640, spp=1),
        # one path bounce of a million rays on a million triangles, an odd count of them alive
        dict(name="bounce_1m", kind="bounce", accel="ray-bvh", scene="spheres", tris=1024000, n=1000003),
        # a small path-traced preview, where the wavefront's launches count
        dict(name="render_preview", kind="render", accel="ray-bvh", scene="terrain", tris=20000, w=211, h=157, spp_x=1, spp_y=1, integrator="path"),
        # direct lighting of an ordinary still with four area-light samples
        dict(name="render_direct", kind="render", accel="ray-bvh", scene="terrain", tris=181250, w=640, h=480, spp_x=2, spp_y=2, integrator="directlighting"),
        # the path-traced frame: 1024 x 1024 at 8 samples, 1,024,000 triangles, depth 5
        dict(name="render_path", kind="render", accel="ray-bvh", scene="spheres", tris=1024000, w=1024, h=1024, spp_x=2, spp_y=4, integrator="path"),
        # 64 scenes of uneven size, mixed camera, path and shadow rays, tuned once as such a program does
        dict(name="set_64", kind="set", scenes=64, median=20000, rays_lo=4096, rays_hi=524288),
        # online training of the learned ordering: 8 SGD steps on 8,192 records
        dict(name="train_8x8192", kind="train", scene="spheres", tris=128000, batch=8192, steps=8),
        # the shadow rays of a frame's camera hits, walked in the learned order
        dict(name="ordered_1m", kind="ordered", scene="spheres", tris=1024000, n=921600),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "tile", "bounce", "bounce", "render", "render", "set", "train", "ordered"])
    if kind == "frame":
        accel = rng.choice(["naive", "rayhierarchy", "ray-bvh"])
        top = 300000 if accel == "naive" else 2000000
        w = _log(rng, 17, 1024)
        spp = rng.choice([1, 1, 2, 4])
        h = max(1, min(_log(rng, 13, 1024), top // (w * spp)))
        return dict(kind=kind, accel=accel, scene="terrain", tris=_log(rng, 1000, 20000 if accel == "naive" else 181250), w=w, h=h, spp=spp,
                    lights=rng.randint(0, 4))
    if kind == "tile":
        accel = rng.choice(["naive", "rayhierarchy", "ray-bvh"])
        return dict(kind=kind, accel=accel, scene="terrain", tris=_log(rng, 1000, 20000 if accel == "naive" else 181250),
                    w=_log(rng, 16, 640), h=_log(rng, 16, 640), spp=1)
    if kind == "bounce":
        return dict(kind=kind, accel="ray-bvh", scene=rng.choice(["terrain", "spheres"]), tris=_log(rng, 2000, 1024000), n=_log(rng, 1000, 1000000))
    if kind == "render":
        accel = rng.choice(["ray-bvh", "ray-bvh", "rayhierarchy", "naive"])
        return dict(kind=kind, accel=accel, scene=rng.choice(["terrain", "spheres"]), tris=_log(rng, 2000, 8000 if accel == "naive" else 1024000 if accel == "ray-bvh" else 181250),
                    w=_log(rng, 24, 200 if accel == "naive" else 800), h=_log(rng, 24, 200 if accel == "naive" else 600),
                    spp_x=rng.randint(1, 2), spp_y=rng.randint(1, 2), integrator=rng.choice(["path", "directlighting"]))
    if kind == "set":
        return dict(kind=kind, scenes=rng.randint(2, 48), median=_log(rng, 2000, 20000), rays_lo=rng.randint(1, 4096), rays_hi=_log(rng, 8192, 262144))
    if kind == "train":
        return dict(kind=kind, scene="spheres", tris=_log(rng, 20000, 256000), batch=512 * rng.randint(1, 16), steps=rng.randint(1, 8))
    return dict(kind=kind, scene=rng.choice(["terrain", "spheres"]), tris=_log(rng, 20000, 1024000), n=_log(rng, 5000, 921600))


# ------------------------------------------------------------------ scenes

@functools.lru_cache(maxsize=None)
def _icosphere(dev):
    v, f = S.icosphere(3)
    return torch.from_numpy(v).to(dev), torch.from_numpy(f).to(dev)


def _spheres(gen, n, center, radius, noise):
    """n icospheres [n * 1280, 3, 3]: vertices pushed in or out by `noise`, turned at random."""
    v, f = _icosphere(str(gen.device))
    disp = 1 + noise * (2 * torch.rand(n, v.shape[0], 1, generator=gen, device=gen.device, dtype=torch.float64) - 1)
    q = torch.randn(n, 4, generator=gen, device=gen.device, dtype=torch.float64)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    rot = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                       2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                       2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1).view(n, 3, 3)
    p = torch.einsum("nvc,nrc->nvr", v[None] * disp, rot) * radius.view(n, 1, 1) + center.view(n, 1, 3)
    return p[:, f].reshape(-1, 3, 3)


def _terrain(gen, tris, extent=16.0, amplitude=2.0):
    """About `tris` triangles: half a six-octave height field, half spheres that stand on it."""
    dev = gen.device
    k = max(1, int(round(tris * (0.5 if tris < 150000 else 0.28) / SPHERE_TRIS)))
    g = max(8, int(round(math.sqrt(max(tris - k * SPHERE_TRIS, 128) / 2))) + 1)
    xs = torch.linspace(-extent / 2, extent / 2, g, device=dev, dtype=torch.float64)
    X, Z = torch.meshgrid(xs, xs, indexing="ij")
    table = torch.rand(256, 256, generator=gen, device=dev, dtype=torch.float64)
    H, amp, freq, norm = torch.zeros_like(X), 1.0, 1.0, 0.0
    for _ in range(6):
        fx, fz = X / extent * 8 * freq, Z / extent * 8 * freq
        ix, iz = torch.floor(fx).long(), torch.floor(fz).long()
        tx, tz = fx - ix, fz - iz
        tx, tz = tx * tx * (3 - 2 * tx), tz * tz * (3 - 2 * tz)
        a, b = table[ix % 256, iz % 256], table[(ix + 1) % 256, iz % 256]
        c, d = table[ix % 256, (iz + 1) % 256], table[(ix + 1) % 256, (iz + 1) % 256]
        H += amp * (2 * ((a * (1 - tx) + b * tx) * (1 - tz) + (c * (1 - tx) + d * tx) * tz) - 1)
        norm, amp, freq = norm + amp, amp * 0.5, freq * 2.0
    H = H * (amplitude / norm)
    P = torch.stack([X, H, Z], -1)
    a, b, c, d = P[:-1, :-1], P[1:, :-1], P[1:, 1:], P[:-1, 1:]
    field = torch.stack([torch.stack([a, c, b], 2), torch.stack([a, d, c], 2)], 2).reshape(-1, 3, 3)
    r = 0.2 + 1.3 * torch.rand(k, generator=gen, device=dev, dtype=torch.float64)
    at = torch.randint(0, g, (2, k), generator=gen, device=dev)
    center = torch.stack([xs[at[0]], H[at[0], at[1]] + r, xs[at[1]]], 1)
    return torch.cat([field, _spheres(gen, k, center, r, 0.0)]).float()


def _boxed(gen, tris, box=40.0):
    """Displaced icospheres of log-uniform size in a box."""
    n = max(1, tris // SPHERE_TRIS)
    r = torch.exp(math.log(0.3) + math.log(10.0) * torch.rand(n, generator=gen, device=gen.device, dtype=torch.float64))
    center = box * (torch.rand(n, 3, generator=gen, device=gen.device, dtype=torch.float64) - 0.5)
    return _spheres(gen, n, center, r, 0.1).float()


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) % (1 << 62))
    return g


VIEW = {"terrain": dict(eye=(0.0, 9.0, -14.0), look=(0.0, 0.0, 0.0), fov=50.0, quad=((-0.5, 12.0, -0.5), (0.5, 12.0, -0.5), (0.5, 12.0, 0.5), (-0.5, 12.0, 0.5))),
        "spheres": dict(eye=(0.0, 6.0, -62.0), look=(0.0, 0.0, 0.0), fov=42.0, quad=((-12.0, 32.0, -12.0), (12.0, 32.0, -12.0), (12.0, 32.0, 12.0), (-12.0, 32.0, 12.0))),
        "sphere": dict(eye=(0.0, 1.0, -4.0), look=(0.0, 0.0, 0.0), fov=45.0, quad=((2.0, 4.0, -2.0),) * 4)}


def _scene(case, gen):
    if case["scene"] == "sphere":
        t = torch.from_numpy(np.concatenate([S.uv_sphere(), S.ground_quad()], 0)).view(-1, 3, 3).to(gen.device)
        turn = float(torch.rand(1, generator=gen, device=gen.device)) * 2 * math.pi
        c, s = math.cos(turn), math.sin(turn)
        t[:-2] = t[:-2] @ torch.tensor([[c, 0, -s], [0, 1, 0], [s, 0, c]], device=gen.device, dtype=torch.float32)
        return t
    return _terrain(gen, case["tris"]) if case["scene"] == "terrain" else _boxed(gen, case["tris"])


# -------------------------------------------------------------------- rays

def _camera(view, w, h, spp, gen, jitter=True):
    """o4, d4 of a pinhole camera's rays in scanline order; the eye is a little off for each seed."""
    dev = gen.device
    eye, _, _, _ = S.look_at(view["eye"], view["look"])
    eye = torch.tensor(eye, device=dev) + 0.05 * (torch.rand(3, generator=gen, device=dev, dtype=torch.float64) - 0.5)
    _, r, u, f = S.look_at(eye.cpu().numpy(), view["look"])
    r, u, f = (torch.tensor(x, device=dev) for x in (r, u, f))
    n = w * h * spp
    pix = torch.arange(w * h, device=dev).repeat_interleave(spp)
    j = torch.rand(2, n, generator=gen, device=dev, dtype=torch.float64) if jitter else torch.full((2, n), 0.5, device=dev, dtype=torch.float64)
    scale, aspect = math.tan(math.radians(view["fov"]) / 2), w / h
    sx = (2 * ((pix % w) + j[0]) / w - 1) * scale * max(aspect, 1.0)
    sy = (1 - 2 * (torch.div(pix, w, rounding_mode="floor") + j[1]) / h) * scale / min(aspect, 1.0)
    d = sx[:, None] * r + sy[:, None] * u + f
    d = d / d.norm(dim=1, keepdim=True)
    o4 = torch.zeros(n, 4, device=dev)
    d4 = torch.full((n, 4), math.inf, device=dev)
    o4[:, :3] = eye.float()
    d4[:, :3] = d.float()
    return o4, d4


def _hits(acc, o4, d4, valid=None):
    n = o4.shape[0]
    out = [torch.empty(n, dtype=torch.int32, device="cuda")] + [torch.empty(n, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    acc.intersect_device(o4, d4, *out, valid=valid)
    torch.cuda.synchronize()
    return out


def _shadow(view, o4, d4, prim, t, gen):
    """Shadow segments from the hits to random points of the light, and which rays have one."""
    hit = prim >= 0
    p = (o4[:, :3] + d4[:, :3] * torch.where(hit, t, torch.zeros_like(t))[:, None]).float()
    q = torch.tensor(view["quad"], device="cuda", dtype=torch.float64)
    uv = torch.rand(2, p.shape[0], generator=gen, device="cuda", dtype=torch.float64)
    d = q[0] + uv[0][:, None] * (q[1] - q[0]) + uv[1][:, None] * (q[3] - q[0]) - p
    dist = d.norm(dim=1).clamp_min(1e-12)
    so = torch.cat([p, torch.where(hit, 1e-3 * t, torch.zeros_like(t))[:, None]], 1).float().contiguous()
    sd = torch.cat([d / dist[:, None], (dist * (1 - 1e-3))[:, None]], 1).float().contiguous()
    return so, sd, hit.to(torch.uint8).contiguous()


def _leave(tris, o4, d4, prim, t, gen):
    """Cosine-weighted directions from the hits, on the side that the ray came from."""
    hit = prim >= 0
    v = tris[prim.clamp_min(0).long()].double()
    nrm = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    nrm = nrm / nrm.norm(dim=1, keepdim=True).clamp_min(1e-30)
    nrm = torch.where((nrm * d4[:, :3]).sum(1, keepdim=True) > 0, -nrm, nrm)
    d = torch.randn(nrm.shape, generator=gen, device="cuda", dtype=torch.float64)
    d = nrm * 1.0001 + d / d.norm(dim=1, keepdim=True).clamp_min(1e-30)
    d = d / d.norm(dim=1, keepdim=True).clamp_min(1e-30)
    n = o4.shape[0]
    bo = torch.zeros(n, 4, device="cuda")
    bd = torch.full((n, 4), math.inf, device="cuda")
    bo[:, :3] = o4[:, :3] + d4[:, :3] * torch.where(hit, t, torch.zeros_like(t))[:, None]
    bo[:, 3] = torch.where(hit, 1e-3 * t, torch.zeros_like(t))
    bd[:, :3] = torch.where(hit[:, None], d, torch.ones_like(d)).float()
    return bo, bd, hit.to(torch.uint8).contiguous()


def _image_of(n):
    """A ray image of at least n pixels, a little wider than high."""
    w = max(1, int(math.ceil(math.sqrt(n * 1.2))))
    return w, -(-n // w)


def _soa(o4, d4):
    return np.ascontiguousarray(torch.cat([o4[:, :3], d4[:, :3], o4[:, 3:], d4[:, 3:]], 1).t().cpu().numpy())


# ----------------------------------------------------------------- prepare

def prepare(case, seed):
    gen = _gen(seed * 1000003 + 17)
    st = {"case": case, "kind": case["kind"]}
    if case["kind"] == "set":
        return _prepare_set(case, gen, st)
    tris = _scene(case, gen)
    view = VIEW[case["scene"]]
    acc = A.MakeAccelerator(case.get("accel", "ray-bvh"), tris.reshape(-1, 9).cpu().numpy())
    st.update(acc=acc, tris=tris)
    if case["kind"] == "render":
        r2c, c2w = R.perspective_camera(case["w"], case["h"], view["eye"], view["look"], (0.0, 1.0, 0.0), view["fov"])
        st["camera"] = R.camera_struct(r2c, c2w, case["w"], case["h"])
        st["lights"] = [R.quad_light(np.asarray(view["quad"], np.float32), (12.0, 12.0, 12.0), 4 if case["integrator"] == "directlighting" else 1)]
        st["params"] = R.render_params(case["integrator"], spp=(case["spp_x"], case["spp_y"]), jitter=True, max_depth=5, seed=seed % 100000 + 1)
    elif case["kind"] in ("frame", "tile"):
        w, h, spp = case["w"], case["h"], case["spp"]
        o4, d4 = _camera(view, w, h, spp, gen, jitter=case["scene"] != "sphere")
        acc.Preprocess(xres=w, yres=h, samplesPerPixel=spp)
        hits = _hits(acc, o4, d4)
        shadows = [_shadow(view, o4, d4, hits[0], hits[1], gen) for _ in range(case.get("lights", 1))]
        if case["kind"] == "frame":
            st.update(o4=o4, d4=d4, shadows=shadows, hits=[torch.empty_like(x) for x in hits], occ=[torch.empty_like(s[2]) for s in shadows])
        else:
            st.update(rays=_soa(o4, d4), shadow=_soa(*shadows[0][:2]), hit=shadows[0][2].bool().cpu().numpy())
    elif case["kind"] in ("bounce", "ordered"):
        n = case["n"]
        w, h = _image_of(n)
        o4, d4 = (x[:n].contiguous() for x in _camera(view, w, h, 1, gen))
        hits = _hits(acc, o4, d4)
        st["shadow"] = _shadow(view, o4, d4, hits[0], hits[1], gen)
        st["occ"] = torch.empty(n, dtype=torch.uint8, device="cuda")
        if case["kind"] == "bounce":
            st["bounce"] = _leave(tris, o4, d4, hits[0], hits[1], gen)
            st["hits"] = [torch.empty_like(x) for x in hits]
        else:
            acc.learn_enable(True, seed=5, queries=2)
            for _ in range(3):  # records from earlier light samples, then the training that a frame ends with
                so, sd, valid = _shadow(view, o4, d4, hits[0], hits[1], gen)
                torch.cuda.synchronize()
                acc.occluded_device(so, sd, st["occ"], valid=valid)
                acc.learn_train(16)
    elif case["kind"] == "train":
        b = case["batch"]
        w, h = _image_of(6 * b)
        o4, d4 = _camera(view, w, h, 1, gen)
        hits = _hits(acc, o4, d4)
        bo, bd, valid = _leave(tris, o4, d4, hits[0], hits[1], gen)
        second = _hits(acc, bo, bd, valid)
        # b rays that hit something: camera rays, and where they are too few bounce rays beside them
        o, d = (torch.cat([x[k >= 0] for x, k in ((p, hits[0]), (q, second[0]))]) for p, q in ((o4, bo), (d4, bd)))
        pick = torch.randperm(o.shape[0], generator=gen, device="cuda")[:b]
        if pick.numel() < b:
            pick = pick.repeat(-(-b // pick.numel()))[:b]
        o, d = o[pick].contiguous(), d[pick].contiguous()
        acc.learn_enable(True, batch=b, records=b, seed=5, queries=1)
        for k in range(4):  # a batch appends at most a quarter of the records kept
            _hits(acc, o[k * b // 4:(k + 1) * b // 4].contiguous(), d[k * b // 4:(k + 1) * b // 4].contiguous())
        st["weights"] = np.zeros(NPARAM, np.float32)
    torch.cuda.synchronize()
    return st


def _prepare_set(case, gen, st):
    n = case["scenes"]
    view = VIEW["terrain"]
    rng = np.random.default_rng(case["median"])  # how uneven the sizes are is the case's, what they hold the seed's
    sizes = np.exp(math.log(case["median"]) + rng.normal(size=n)).clip(1000, 500000).astype(int).tolist()
    rays = rng.integers(case["rays_lo"], case["rays_hi"] + 1, n).tolist()
    scenes, near, shadow = [], [], []
    for size, m in zip(sizes, rays):
        tris = _terrain(gen, size)
        scenes.append(tris.reshape(-1, 9).cpu().numpy())
        cam, path = int(m * 0.4), int(m * 0.3)
        w, h = _image_of(max(cam, 1))
        o4, d4 = (x[:cam] for x in _camera(view, w, h, 1, gen))
        # points all over the surface, which path and shadow rays leave
        at = torch.randint(0, tris.shape[0], (m - cam,), generator=gen, device="cuda")
        uv = torch.rand(2, m - cam, generator=gen, device="cuda")
        s = uv[0].sqrt()
        v = tris[at]
        p = (1 - s)[:, None] * v[:, 0] + (s * (1 - uv[1]))[:, None] * v[:, 1] + (s * uv[1])[:, None] * v[:, 2]
        nrm = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
        nrm = nrm / nrm.norm(dim=1, keepdim=True).clamp_min(1e-30)
        nrm = torch.where(nrm[:, 1:2] < 0, -nrm, nrm)
        p = p + 1e-3 * nrm
        po = torch.zeros(path, 4, device="cuda")
        pd = torch.full((path, 4), math.inf, device="cuda")
        d = torch.randn(path, 3, generator=gen, device="cuda")
        d = nrm[:path] * 1.0001 + d / d.norm(dim=1, keepdim=True).clamp_min(1e-30)
        po[:, :3], pd[:, :3] = p[:path], d / d.norm(dim=1, keepdim=True).clamp_min(1e-30)
        q = p[path:]
        fake = torch.zeros(q.shape[0], dtype=torch.int32, device="cuda")
        q4 = torch.cat([q, torch.zeros_like(q[:, :1])], 1)
        so, sd, _ = _shadow(view, q4, torch.zeros_like(q4), fake, torch.ones(q.shape[0], device="cuda"), gen)
        near.append((torch.cat([o4, po]), torch.cat([d4, pd])))
        shadow.append((so, sd))
    st["set"] = B.SceneSet(scenes)
    a = {}
    for key, parts in (("n", near), ("s", shadow)):
        a["o4" + key] = torch.cat([x[0] for x in parts]).contiguous()
        a["d4" + key] = torch.cat([x[1] for x in parts]).contiguous()
        a[{"n": "near_offsets", "s": "occ_offsets"}[key]] = np.concatenate([[0], np.cumsum([x[0].shape[0] for x in parts])]).astype(np.int64)
    k = a["o4n"].shape[0]
    a["prim"] = torch.empty(k, dtype=torch.int32, device="cuda")
    for key in ("t", "b1", "b2"):
        a[key] = torch.empty(k, device="cuda")
    a["occ"] = torch.empty(a["o4s"].shape[0], dtype=torch.uint8, device="cuda")
    st["args"] = a
    st["tuned"] = st["set"].autotune(**a)
    torch.cuda.synchronize()
    return st


# --------------------------------------------------------------------- run

def run(st):
    kind, acc = st["kind"], st.get("acc")
    if kind == "frame":
        acc.intersect_device(st["o4"], st["d4"], *st["hits"])
        for (so, sd, valid), occ in zip(st["shadows"], st["occ"]):
            acc.occluded_device(so, sd, occ, valid=valid)
        return [*st["hits"], *st["occ"]]
    if kind == "tile":
        rays = st["rays"]
        rays[7] = np.inf  # fresh camera rays: Intersect leaves each hit's t there
        prim, t, b1, b2 = acc.Intersect(rays)
        geo = acc.HitGeometry(rays, prim, t, b1, b2)
        occ = acc.IntersectP(st["shadow"], hit=st["hit"])
        return [prim, t, b1, b2, geo, occ]
    if kind == "bounce":
        bo, bd, valid = st["bounce"]
        acc.intersect_device(bo, bd, *st["hits"], valid=valid)
        so, sd, valid = st["shadow"]
        acc.occluded_device(so, sd, st["occ"], valid=valid)
        return [*st["hits"], st["occ"]]
    if kind == "render":
        img, _ = R.render(acc, st["camera"], st["lights"], st["params"])
        return img
    if kind == "set":
        a = st["args"]
        st["set"].trace(**a)
        return [a["prim"], a["t"], a["b1"], a["b2"], a["occ"]]
    if kind == "train":
        acc.learn_train(st["case"]["steps"])
        lib = L.lib()
        L.check(lib.pbg_learn_params_io(acc.handle, C.c_void_p(st["weights"].ctypes.data), C.c_int32(1)), "pbg_learn_params_io")
        return st["weights"]
    so, sd, valid = st["shadow"]
    acc.occluded_device(so, sd, st["occ"], valid=valid)
    return st["occ"]


# -------------------------------------------------------------------- work

RAY, HIT = 32, 16  # bytes of a ray record and of a hit's prim, t, b1, b2
TEST = 45          # operations of one exact ray/triangle test


def _walk(n, tris):
    """Operations of n walks: a box test (12) on each level of a binary tree over the triangles, and one triangle test."""
    return n * (12.0 * math.log2(max(tris, 2)) + TEST)


def work(case):
    kind, tris = case["kind"], case.get("tris", 0)
    if kind in ("frame", "tile"):
        n, m = case["w"] * case["h"] * case["spp"], case.get("lights", 1)
        geo = 56 if kind == "tile" else 0
        return {"bytes": n * (RAY + HIT + geo) + n * m * (RAY + 2) + 36 * tris, "flops": _walk(n * (1 + m), tris)}
    if kind == "bounce":
        return {"bytes": case["n"] * (RAY + 1 + HIT + RAY + 2) + 36 * tris, "flops": _walk(2 * case["n"], tris)}
    if kind == "render":
        pix = case["w"] * case["h"]
        n = pix * case["spp_x"] * case["spp_y"]
        # direct lighting: the camera ray and four shadow rays; path: about as many again over its bounces
        return {"bytes": 12 * pix + 36 * tris, "flops": _walk(n * (5 if case["integrator"] == "directlighting" else 4), tris)}
    if kind == "set":
        n = case["scenes"] * (case["rays_lo"] + case["rays_hi"]) / 2
        tris = case["median"] * math.exp(0.5)
        return {"bytes": n * (RAY + 0.7 * HIT + 0.3) + 36 * tris * case["scenes"], "flops": _walk(n, tris)}
    if kind == "train":
        mac = 112 * 64 + 64 * 64 + 64 * 256
        return {"bytes": case["steps"] * case["batch"] * (112 * 2 + 4) + 8 * NPARAM, "flops": 6.0 * case["steps"] * case["batch"] * mac}
    mac = 112 * 64 + 64 * 64 + 64 * 256
    return {"bytes": case["n"] * (RAY + 2) + 36 * tris, "flops": 2.0 * case["n"] * mac + _walk(case["n"], tris)}


# ------------------------------------------------------------------- exact

def _nearest64(tris, o4, d4, valid=None):
    """t, b1, b2 of each ray's nearest hit, every triangle tried, in 64 bits (misses: zeros)."""
    v = tris.double()
    p1, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    out = torch.zeros(3, o4.shape[0], device=o4.device, dtype=torch.float64)
    step = max(1, (1 << 23) // max(1, v.shape[0]))
    cross = lambda a, b: (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])  # noqa: E731
    dot = lambda a, b: a[0] * b[0] + a[1] * b[1] + a[2] * b[2]  # noqa: E731
    P, E1, E2 = ([x[:, k][None] for k in range(3)] for x in (p1, e1, e2))
    for k in range(0, o4.shape[0], step):
        o, d = o4[k:k + step].double(), d4[k:k + step].double()
        O, D = ([x[:, j][:, None] for j in range(3)] for x in (o, d))
        s1 = cross(D, E2)
        inv = 1.0 / dot(s1, E1)
        V = [a - b for a, b in zip(O, P)]
        b1 = dot(V, s1) * inv
        s2 = cross(V, E1)
        b2 = dot(D, s2) * inv
        t = dot(E2, s2) * inv
        ok = torch.isfinite(inv) & (b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t >= o[:, 3:]) & (t <= d[:, 3:])
        if valid is not None:
            ok &= valid[k:k + step, None] != 0
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        best, at = t.min(1)
        hit = torch.isfinite(best)
        pick = lambda x: torch.where(hit, x.gather(1, at[:, None])[:, 0], torch.zeros_like(best))  # noqa: E731
        out[0, k:k + step] = torch.where(hit, best, torch.zeros_like(best))
        out[1, k:k + step], out[2, k:k + step] = pick(b1), pick(b2)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("frame", "tile", "bounce"):
        return None  # an image, many scenes' hits, weights whose labels are the framework's own clusters, or bytes only
    n = case["n"] if kind == "bounce" else case["w"] * case["h"] * case["spp"]
    if n * case["tris"] > 1.5e10:
        return None
    st = prepare(case, seed)
    tris = st["tris"]
    if kind == "frame":
        return [None, *_nearest64(tris, st["o4"], st["d4"]), *([None] * case["lights"])]
    if kind == "bounce":
        return [None, *_nearest64(tris, *st["bounce"]), None]
    r = torch.from_numpy(st["rays"]).cuda()
    r[7] = math.inf
    o4, d4 = torch.stack([r[0], r[1], r[2], r[6]], 1), torch.stack([r[3], r[4], r[5], r[7]], 1)
    t, b1, b2 = _nearest64(tris, o4, d4)
    prim = _hits(st["acc"], o4.contiguous(), d4.contiguous())[0]  # which triangle: its geometry below is plain 64-bit arithmetic
    v = tris[prim.clamp_min(0).long()].double()
    p = o4[:, :3].double() + d4[:, :3].double() * t[:, None]
    du, dv = v[:, 1] - v[:, 0], v[:, 2] - v[:, 1]  # of the default uvs (0,0), (1,0), (1,1)
    nn = torch.linalg.cross(du, dv)
    nn = nn / nn.norm(dim=1, keepdim=True).clamp_min(1e-300)
    geo = torch.cat([p, du, dv, nn, (b1 + b2)[:, None], b2[:, None]], 1)
    geo = torch.where((prim >= 0)[:, None], geo, torch.zeros_like(geo))
    return [None, t, b1, b2, geo, None]
