"""What a program does with this renderer, as cases that can be timed.

A case is a dict of plain values.  `listed()` gives the ones that stand for
the renderer's uses, `draw(rng)` one more of the same ranges, `prepare(case,
seed)` what a program has in hand before the call (the scene loaded, inputs on
the GPU), `run(state)` one pass through the public entry points, `work(case)`
the bytes and operations a pass cannot do without, and `exact(case, seed)` the
results in 64 bits where plain torch gives them in reasonable time.

Kinds of case:
  cast       closest hits of a program's own rays (GpuRenderer.cast_rays)
  ids        object and triangle ids of a frame's primary rays (primary_hits)
  gather     estimates of a photon map at given points (photon_gather)
  bake       photon maps shot, then both estimated at given points
  frame      a whole frame (render): acceleration structures, photons, pixels
  batch      several frames in one wavefront (render_batch)
  infer      the radiance-cache network on given samples (RadianceCache.infer)
  gradients  its loss and gradient over a batch of samples

The scenes are the benchmark's (sray_gb300/scenegen.py): `terrain` (a
displaced grid of nx * nz * 2 triangles with instanced spheres of triangles,
three sphere lights), `small` (5,122 triangles, quadrics, a point light) and
`movers` (a terrain with spheres moving on keyframes, motion blur).  A process
holds one renderer; it is loaded when a case first needs its scene and kept.
"""
import math
import re

import numpy as np
import torch

from sray_gb300 import scenegen
from sray_gb300.gpu import GpuRenderer, RadianceCache

N_PARAMS = 26563                                   # the network's parameters
NET = [(64, 216), (64, 64), (64, 64), (64, 64), (3, 64)]
SAMPLE_FLOPS = 2 * sum(o * i for o, i in NET)      # multiply-adds of one sample, twice


def listed():
    return [
        # picking with a pointer, probing a few lines of sight: a handful of rays, the latency counts
        dict(name="pick", kind="cast", scene="terrain", nx=1000, nz=500, rays=64),
        # ambient occlusion and visibility of a light map: a million rays that head everywhere
        dict(name="visibility", kind="cast", scene="terrain", nx=1000, nz=500, rays=1000003),
        # light map of the production scene: its photon maps shot anew, then estimated at every texel
        dict(name="bake", kind="bake", scene="terrain", nx=1000, nz=500, caust=500000, gi=2000000, points=200001),
        # the production still at full size, four samples a pixel, with its 2.5M photons
        dict(name="still", kind="frame", scene="terrain", nx=1000, nz=500, width=1920, height=1080, smin=4, smax=4,
             caust=500000, gi=2000000),
        # object and depth buffers of a moving scene for compositing, full size
        dict(name="ids", kind="ids", scene="movers", tris=100000, width=1920, height=1080),
        # a short stretch of animation in one wavefront, motion-blurred
        dict(name="animation", kind="batch", scene="movers", tris=100000, frames=6, width=480, height=270, smin=2, smax=2,
             caust=20000, gi=80000),
        # a draft of the production settings (1-16 samples by variance) at an odd size
        dict(name="draft", kind="frame", scene="movers", tris=100000, width=321, height=181, smin=1, smax=16,
             caust=20000, gi=80000),
        # the interactive preview: one sample a pixel of the small scene, few photons
        dict(name="preview", kind="frame", scene="small", width=320, height=240, smin=1, smax=1, caust=20000, gi=0),
        # probes placed in the scene: a few estimates per call
        dict(name="probes", kind="gather", scene="small", which=1, k=100, caust=100000, gi=500000, points=200),
        # irradiance of a whole light map from the k nearest photons
        dict(name="irradiance", kind="gather", scene="small", which=1, k=100, caust=100000, gi=500000, points=500009),
        # the radiance cache's queries of a 4K frame and its training step
        dict(name="cache queries", kind="infer", samples=4194304),
        dict(name="cache training", kind="gradients", samples=16384),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cast", "cast", "ids", "gather", "gather", "bake", "frame", "frame", "batch", "infer", "gradients"])
    terrain = rng.choice([dict(nx=60, nz=30), dict(nx=300, nz=150), dict(nx=1000, nz=500)])
    tris = rng.choice([12000, 100000, 400000])
    if kind == "infer":
        return dict(kind=kind, samples=_log(rng, 100, 4000000))
    if kind == "gradients":
        return dict(kind=kind, samples=_log(rng, 64, 262144))
    if kind == "cast":
        scene = rng.choice(["terrain", "movers", "small"])
        c = dict(kind=kind, scene=scene, rays=_log(rng, 16, 1000000))
        c.update(terrain if scene == "terrain" else dict(tris=tris) if scene == "movers" else {})
        return c
    if kind == "gather":
        photons = _log(rng, 20000, 500000)
        return dict(kind=kind, scene="small", which=rng.choice([0, 1]), k=rng.choice([0, 50, 100]), caust=photons // 2 + 1,
                    gi=photons, points=_log(rng, 16, 500000))
    if kind == "bake":
        photons = _log(rng, 20000, 2000000)
        return dict(kind=kind, scene="terrain", caust=photons // 4, gi=photons, points=_log(rng, 100, 200000), **terrain)
    if kind == "ids":
        w = _log(rng, 64, 1900)
        return dict(kind=kind, scene="movers", tris=tris, width=w, height=max(16, int(w * rng.uniform(0.4, 0.56))))
    if kind == "batch":
        w = _log(rng, 64, 480)
        s = rng.choice([1, 2])
        return dict(kind=kind, scene="movers", tris=tris, frames=rng.randint(2, 6), width=w, height=max(16, int(w * rng.uniform(0.5, 0.6))),
                    smin=s, smax=s, caust=_log(rng, 2000, 20000), gi=_log(rng, 8000, 80000))
    scene = rng.choice(["terrain", "movers", "small"])
    w = _log(rng, 64, 1900)
    smin, smax = (1, 16) if w <= 480 and rng.random() < 0.4 else rng.choice([(1, 1), (2, 2), (4, 4)])
    photons = _log(rng, 4000, 2000000)
    c = dict(kind="frame", scene=scene, width=w, height=max(16, int(w * rng.uniform(0.4, 0.56))), smin=smin, smax=smax,
             caust=photons // 4, gi=0 if scene == "small" and rng.random() < 0.5 else photons)
    c.update(terrain if scene == "terrain" else dict(tris=tris) if scene == "movers" else {})
    return c


# ---- the process's renderer ----

_held = {}     # "g": the renderer, "scene": what it has loaded, "opts": its options, "ready": what is built


def _scene_file(case):
    if case["scene"] == "terrain":
        return scenegen.write_scene("production", grid=(case["nx"], case["nz"]), n_inst=200 if case["nx"] >= 1000 else 40)
    if case["scene"] == "movers":
        return scenegen.write_scene("batch", seed=1000, tris=case["tris"])
    return scenegen.write_scene("small")


def _options(case):
    o = scenegen.scene_opts("small" if case["scene"] == "small" else "production")
    if case["scene"] == "movers":
        o.update(mblur=1, shutter=8)
    o.update(width=case.get("width", 1920), height=case.get("height", 1080), min_samples=case.get("smin", 1),
             max_samples=case.get("smax", 1), caust_photons=case.get("caust", 0), gi_photons=case.get("gi", 0))
    if case["scene"] == "small":
        o.update(gi_k=100)
    if "k" in case:
        # k = 0: every photon within a fixed radius, as the scene's default options gather
        o.update(caust_k=case["k"], gi_k=case["k"], gather_dist=0.01)
    return o


def _renderer(case):
    opts = _options(case)
    scene = (_scene_key(case), opts["width"], opts["height"], opts["meshoct_max_depth"], opts.get("shutter", 0))
    if _held.get("scene") != scene:
        if "g" in _held:
            _held["g"].close()
            _held.clear()
        g = GpuRenderer(**opts)
        g.load(_scene_file(case))
        _held.update(g=g, scene=scene, opts=opts, ready="")
    g = _held["g"]
    if _held["opts"] != opts:
        g.set_opts(**opts)
        _held.update(opts=opts, ready="")
    if case["kind"] in ("cast", "gather") and _held["ready"] != case["kind"]:
        # a program builds once and then asks many times
        g.build(0, 8 if case["scene"] == "movers" else 0)
        if case["kind"] == "gather":
            g.shoot_photons(0, 0)
        _held["ready"] = case["kind"]
    return g


def _scene_key(case):
    return (case["scene"], case.get("nx", 0), case.get("nz", 0), case.get("tris", 0))


def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7fffffffffff)
    return g


def _u(gen, n, lo, hi):
    return torch.rand(n, generator=gen, device="cuda", dtype=torch.float32) * (hi - lo) + lo


def _directions(gen, n):
    d = torch.randn((n, 3), generator=gen, device="cuda", dtype=torch.float32)
    return d / d.norm(dim=1, keepdim=True).clamp_min(1e-6)


def _weights():
    """The network a program has stored: He-uniform weights, small biases."""
    rng = np.random.default_rng(11)
    p = []
    for o, i in NET:
        lim = math.sqrt(6.0 / i)
        p += [rng.uniform(-lim, lim, o * i), rng.uniform(-0.05, 0.05, o)]
    return np.concatenate(p).astype(np.float32)


def _samples(case, seed):
    """Path vertices as the renderer feeds them: position in the unit box,
    normal and incident direction mapped to [0, 1], and radiance targets."""
    n = case["samples"]
    gen = _gen(seed, 3)
    x = torch.cat([_u(gen, (n, 3), 0.0, 1.0), _directions(gen, n) * 0.5 + 0.5, _directions(gen, n) * 0.5 + 0.5], 1).contiguous()
    t = torch.rand((n, 3), generator=gen, device="cuda", dtype=torch.float32) ** 3 * 2.0
    return x, t


def _rays(case, seed):
    """Rays of a program's own: from points over the scene's floor, heading everywhere."""
    n = case["rays"]
    gen = _gen(seed, 1)
    ext = dict(terrain=(45.0, 22.0, -1.0, 12.0), movers=(35.0, 17.0, -1.0, 12.0), small=(9.0, 9.0, 0.1, 6.0))[case["scene"]]
    o = torch.stack([_u(gen, n, -ext[0], ext[0]), _u(gen, n, ext[2], ext[3]), _u(gen, n, -ext[1], ext[1])], 1).contiguous()
    d = (_directions(gen, n) * 200.0).contiguous()
    time = torch.randint(0, 9, (n,), generator=gen, device="cuda", dtype=torch.int32) if case["scene"] == "movers" else None
    return o, d, time


def _points(case, seed, photons):
    """Surface points near where photons landed, with the surfaces' normals."""
    n = case["points"]
    gen = _gen(seed, 2)
    i = torch.randint(0, photons.shape[0], (n,), generator=gen, device="cuda")
    pos = photons[i, 0:3] + (torch.rand((n, 3), generator=gen, device="cuda") - 0.5) * 0.05
    return pos.contiguous(), photons[i, 6:9].contiguous()


def _map_photons(g, which):
    return torch.from_numpy(np.ascontiguousarray(g.photons(which)[:, :13])).cuda()


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, kind=kind, seed=(int(seed) * 2654435761 + 12345) & 0x7fffffffffffffff)
    if kind in ("infer", "gradients"):
        if _held.get("net") is None:
            _held["net"] = RadianceCache(seed=None)
            _held["net"].set_params(_weights())
        st["x"], st["t"] = _samples(case, seed)
        n = case["samples"]
        st["y"] = torch.empty((n, 3), dtype=torch.float32, device="cuda")
        st["grad"] = torch.empty(N_PARAMS, dtype=torch.float32, device="cuda")
        st["loss"] = torch.empty(1, dtype=torch.float32, device="cuda")
        return st
    g = _renderer(case)
    i32 = dict(dtype=torch.int32, device="cuda")
    f32 = dict(dtype=torch.float32, device="cuda")
    if kind in ("cast", "ids"):
        n = case["rays"] if kind == "cast" else case["width"] * case["height"]
        if kind == "cast":
            st["o"], st["d"], st["time"] = _rays(case, seed)
        else:
            st["msec"] = 4 + int(seed) * 37 % 953
        st.update(obj=torch.empty(n, **i32), prim=torch.empty(n, **i32), t=torch.empty(n, **f32),
                  tie=torch.empty(n, dtype=torch.uint8, device="cuda"))
    elif kind == "gather":
        if _held.get("photons_of") != (case["which"], _held["scene"], str(_held["opts"])):
            _held["photons"] = _map_photons(g, case["which"])
            _held["photons_of"] = (case["which"], _held["scene"], str(_held["opts"]))
        st["pos"], st["norm"] = _points(case, seed, _held["photons"])
        st["out"] = torch.empty((case["points"], 3), **f32)
    elif kind == "bake":
        # texels over the terrain: points above its floor, normals mostly up
        n = case["points"]
        gen = _gen(seed, 4)
        st["pos"] = torch.stack([_u(gen, n, -45.0, 45.0), _u(gen, n, -1.0, 1.5), _u(gen, n, -22.0, 22.0)], 1).contiguous()
        st["norm"] = torch.nn.functional.normalize(_directions(gen, n) * 0.3 + torch.tensor([0.0, 1.0, 0.0], device="cuda"), dim=1).contiguous()
        st["out"] = [torch.empty((n, 3), **f32) for _ in range(2)]
    elif kind == "frame":
        st["msec"] = 4 + int(seed) * 37 % 953 if case["scene"] == "movers" else 0
        st["fb"] = torch.zeros((case["height"], case["width"], 4), **f32)
    elif kind == "batch":
        st["msec"] = 4 + int(seed) * 37 % 700
        st["fbs"] = [torch.zeros((case["height"], case["width"], 4), **f32) for _ in range(case["frames"])]
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "infer":
        _held["net"].infer(st["x"], st["y"])
        return st["y"]
    if kind == "gradients":
        _held["net"].gradients(st["x"], st["t"], st["grad"], st["loss"])
        return dict(grad=st["grad"], loss=st["loss"])
    g = _held["g"]
    if kind == "cast":
        g.cast_rays(st["o"], st["d"], st["time"], st["obj"], st["prim"], st["t"], st["tie"])
        return dict(obj=st["obj"], prim=st["prim"], t=st["t"], tie=st["tie"])
    if kind == "ids":
        g.primary_hits(st["obj"], st["prim"], st["t"], st["tie"], msec=st["msec"])
        return dict(obj=st["obj"], prim=st["prim"], t=st["t"], tie=st["tie"])
    if kind == "gather":
        g.photon_gather(case["which"], st["pos"], st["norm"], st["out"])
        return st["out"]
    # the random streams of a frame or a bake are its own
    g.set_opts(seed=st["seed"])
    if kind == "bake":
        stored = g.shoot_photons(0, 0)
        for which in (0, 1):
            g.photon_gather(which, st["pos"], st["norm"], st["out"][which])
        return dict(caustic=st["out"][0], indirect=st["out"][1], stored=list(stored))
    if kind == "frame":
        return g.render(st["msec"], st["fb"])
    g.render_batch([(st["msec"] + 40 * i, fb) for i, fb in enumerate(st["fbs"])])
    return st["fbs"]


def _triangles(case):
    if case["scene"] == "terrain":
        return 2 * case["nx"] * case["nz"] + (200 if case["nx"] >= 1000 else 40) * 1280
    return case["tris"] if case["scene"] == "movers" else 5122


def work(case):
    """Inputs read once, outputs written once; a ray's or a photon's own path
    depends on the scene and is not counted.  A frame reads its scene's
    vertices once (36 bytes a triangle)."""
    kind = case["kind"]
    if kind == "infer":
        return dict(bytes=case["samples"] * 48 + N_PARAMS * 4, flops=case["samples"] * SAMPLE_FLOPS)
    if kind == "gradients":
        return dict(bytes=case["samples"] * 60 + 2 * N_PARAMS * 4, flops=3 * case["samples"] * SAMPLE_FLOPS)
    if kind == "cast":
        return dict(bytes=case["rays"] * (24 + (4 if case["scene"] == "movers" else 0) + 13), flops=0)
    if kind == "ids":
        return dict(bytes=case["width"] * case["height"] * 13 + _triangles(case) * 36, flops=0)
    if kind == "gather":
        return dict(bytes=case["points"] * 36, flops=0)
    if kind == "bake":
        return dict(bytes=case["points"] * 48 + _triangles(case) * 36, flops=0)
    return dict(bytes=case.get("frames", 1) * case["width"] * case["height"] * 16 + _triangles(case) * 36, flops=0)


# ---- the results in 64 bits ----

def _features(x):
    a = math.pi * x.double()[:, :, None] * (2.0 ** torch.arange(12, device=x.device, dtype=torch.float64))
    return torch.stack([torch.sin(a), torch.cos(a)], 3).reshape(x.shape[0], 216)


def _net64():
    p = torch.from_numpy(_weights()).cuda().double()
    ws, o = [], 0
    for r, c in NET:
        ws += [p[o:o + r * c].reshape(r, c), p[o + r * c:o + r * c + r]]
        o += r * c + r
    return ws


def _forward64(ws, x):
    h = _features(x)
    for l in range(5):
        h = h @ ws[2 * l].T + ws[2 * l + 1]
        if l < 4:
            h = h.relu()
    return h


def _exact_net(case, seed):
    x, t = _samples(case, seed)
    ws = _net64()
    if case["kind"] == "infer":
        return torch.cat([_forward64(ws, c) for c in x.split(131072)])
    for w in ws:
        w.requires_grad_(True)
    loss = torch.zeros((), dtype=torch.float64, device="cuda")
    for xc, tc in zip(x.split(32768), t.split(32768)):
        y = _forward64(ws, xc)
        part = (((y - tc.double()) ** 2) / (y.detach() ** 2 + 0.01)).sum() / (3 * case["samples"])
        part.backward()
        loss += part.detach()
    return dict(grad=torch.cat([w.grad.reshape(-1) for w in ws]), loss=loss.reshape(1))


def _world_triangles(path):
    """The scene document's meshes as world-space triangles in 64 bits: [n, 3, 3]."""
    with open(path) as f:
        text = f.read()
    out = []
    for body in re.findall(r'<object type="mesh".*?</object>', text, re.S):
        v = np.array(" ".join(re.findall(r'<vertex id="\d+" val="([^"]*)"', body)).split(), np.float64).reshape(-1, 3)
        f = np.array(re.findall(r'<vref vertex="(\d+)"', body)).astype(np.int64).reshape(-1, 3)
        xf = re.search(r"<xform[^>]*>", body)
        if xf:
            a = {k: np.array(s.split(), np.float64) for k, s in re.findall(r'(\w+)="([^"]*)"', xf.group(0))}
            v = v * a.get("scale", np.ones(3))
            if "axisrot" in a:
                w, u = math.radians(a["axisrot"][0]), a["axisrot"][1:] / np.linalg.norm(a["axisrot"][1:])
                v = v * math.cos(w) + np.cross(u, v) * math.sin(w) + np.outer(v @ u, u) * (1.0 - math.cos(w))
            v = v + a.get("pos", np.zeros(3))
        out.append(v[f])
    return np.concatenate(out)


def _exact_cast(case, seed):
    o, d, _ = _rays(case, seed)
    o, d = o.double(), d.double()
    tris = torch.from_numpy(_world_triangles(_scene_file(case))).cuda()
    best = torch.full((case["rays"],), math.inf, dtype=torch.float64, device="cuda")
    for part in tris.split(max(1, (1 << 23) // case["rays"])):
        a, e1, e2 = part[:, 0], part[:, 1] - part[:, 0], part[:, 2] - part[:, 0]
        p = torch.linalg.cross(d[:, None, :], e2[None, :, :])
        det = (e1[None] * p).sum(-1)
        s = o[:, None, :] - a[None]
        u = (s * p).sum(-1) / det
        q = torch.linalg.cross(s, e1[None].expand_as(s))
        w = (d[:, None, :] * q).sum(-1) / det
        t = (e2[None] * q).sum(-1) / det
        hit = (det != 0) & (u >= 0) & (w >= 0) & (u + w <= 1) & (t >= 1e-6) & (t <= 1)
        best = torch.minimum(best, torch.where(hit, t, math.inf).amin(1))
    return dict(obj=None, prim=None, t=torch.where(torch.isfinite(best), best, 0.0), tie=None)


def _exact_gather(case, seed):
    """The estimate at each point over the stored photons: the k nearest
    within the radius (all of them where k is 0), their power over the area of
    the disc that holds them; fewer than eight caustic photons give none."""
    prepare(case, seed)          # the map's photons are this case's input
    ph = _held["photons"].double()
    pos, norm = _points(case, seed, _held["photons"])
    pos, norm = pos.double(), norm.double()
    k, rad = case["k"], 0.5
    if k == 0:
        return None              # the radius is the scene's own
    out = []
    for q, n in zip(pos.split(max(1, (1 << 25) // ph.shape[0])), norm.split(max(1, (1 << 25) // ph.shape[0]))):
        d2 = ((q[:, None, :] - ph[None, :, 0:3]) ** 2).sum(-1)
        d2 = torch.where(d2 <= rad * rad, d2, math.inf)
        near, idx = torch.topk(d2, min(k, ph.shape[0]), dim=1, largest=False)
        got = torch.isfinite(near)
        cnt = got.sum(1)
        reach = torch.where(got, near, 0.0).amax(1)
        p = ph[idx]
        dirs = -(p[:, :, 3:6] * n[:, None, :]).sum(-1)
        if case["which"] == 0:
            wgt = (got & (dirs > 0)).double()
        else:
            facing = (p[:, :, 6:9] * n[:, None, :]).sum(-1) > math.cos(math.pi / 2.5)
            wgt = torch.where(got & (dirs > 0) & facing, dirs, 0.0)
        est = (p[:, :, 9:12] * wgt[:, :, None]).sum(1) / (math.pi * reach)[:, None]
        out.append(torch.where((cnt >= (8 if case["which"] == 0 else 1))[:, None], est, 0.0))
    return torch.cat(out)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("infer", "gradients"):
        return _exact_net(case, seed)
    if kind == "cast" and case["scene"] == "terrain" and case["rays"] * _triangles(case) <= 400_000_000:
        return _exact_cast(case, seed)
    if kind == "gather" and case["points"] * case["gi"] <= 4_000_000_000:
        return _exact_gather(case, seed)
    return None
