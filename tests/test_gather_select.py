"""The photon gather's selection of the k nearest against double arithmetic.

Photon maps are restored from dumps written here, so that the candidates of
each query are known: none, fewer than k, exactly k, one more, lists at the
edges of a warp (31-33) and of the on-chip list (511-513), more candidates
than the list holds, hundreds of photons at one distance, neighbours one
float apart at the k-th place, and photons just inside and outside the radius.

Bound: an estimate is a sum of at most ~2,000 positive terms, 2,000 / 32 per
lane and five levels over the lanes, each addition and the three roundings of
a term and of the area within 2^-24: (63 + 5 + 6) 2^-24 = 4.4e-6.
"""
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

BOUND = 5e-6


def _layouts():
    rng = np.random.default_rng(7)
    q = np.float64([[-12.0, 1.0, -12.0]])

    def disc(n, lo=0.0, hi=0.49):
        d = np.sqrt(rng.uniform(lo * lo, hi * hi, n))
        a = rng.uniform(0, 2 * np.pi, n)
        return np.stack([d * np.cos(a), rng.uniform(-0.01, 0.01, n), d * np.sin(a)], 1)

    def axis(n, a):
        c = np.float64([[a, 0, 0], [-a, 0, 0], [0, 0, a], [0, 0, -a]])
        return c[np.arange(n) % 4]

    f = np.float32(0.375)
    near = [float(f)]
    for _ in range(5):
        f = np.nextafter(f, np.float32(1))
        near.append(float(f))
    edge = np.float64([[0.5, 0, 0], [0, 0, -0.5], [0.500001, 0, 0], [0, 0, 0.499999], [0.3, 0, 0.4], [0.300001, 0, 0.4]])
    out = {"none": axis(40, 0.75), "one": axis(1, 0.25), "edge": np.concatenate([edge, disc(12)]),
           "at the query": np.zeros((20, 3)), "sphere": rng.normal(size=(1500, 3)) * 0.2,
           "equal 40": np.concatenate([axis(40, 0.25), disc(20, 0.0, 0.2)]),
           "equal 300": np.concatenate([axis(300, 0.25), disc(30, 0.0, 0.2), disc(30, 0.3, 0.4)]),
           "equal 900": np.concatenate([axis(900, 0.25), disc(30, 0.0, 0.2)]),
           "floats apart": np.concatenate([np.float64([[x, 0, 0] for x in near]), disc(47, 0.0, 0.3), disc(20, 0.4, 0.45)]),
           "clustered": np.concatenate([disc(400, 0.0, 0.002), disc(200, 0.0, 0.45)])}
    for n in (7, 8, 31, 32, 33, 49, 50, 51, 64, 65, 511, 512, 513, 700, 2000):
        out["disc %d" % n] = disc(n)
    centres = {name: q[0] + np.float64([2.0 * (i % 6), 0.0, 2.0 * (i // 6)]) for i, name in enumerate(out)}
    return {name: (centres[name], centres[name] + off) for name, off in out.items()}


def _expected(pos, power, q, k, kind, rad):
    """The estimate in double over float positions (PhotonMap::irradiance_est
    and radiance_est with the k nearest within rad, or all within rad for k = 0)."""
    d = pos.astype(np.float64) - np.float32(q).astype(np.float64)
    d2 = (d * d).sum(1)
    ok = d2 <= float(np.float32(rad)) ** 2
    if not ok.any():
        return np.zeros(3)
    key = d2.astype(np.float32)
    if k > 0:
        kth = np.sort(key[ok])[min(k, ok.sum()) - 1]
        ok &= key <= kth
        area = np.pi * float(kth)
    if kind == 0 and ok.sum() < 8:
        return np.zeros(3)
    with np.errstate(divide="ignore", invalid="ignore"):
        return power[ok].astype(np.float64).sum(0) / (area if k > 0 else np.pi * rad ** 2)


@pytest.fixture(scope="module")
def dump(tmp_path_factory):
    """one dump of every layout's photons, in any order"""
    lay = _layouts()
    rng = np.random.default_rng(8)
    pos = np.concatenate([p for _, p in lay.values()])
    pos = pos[rng.permutation(len(pos))]
    power = rng.uniform(0.5, 2.0, (len(pos), 3))
    path = os.path.join(str(tmp_path_factory.mktemp("dump")), "photons")
    with open(path, "w") as f:
        f.write("energy 300.0\n")
        for p, c in zip(pos, power):
            f.write("<%.6f %.6f %.6f> <0.0 -1.0 0.0> <0.0 1.0 0.0> <%.6f %.6f %.6f>\n" % (*p, *c))
    as_read = [np.array([[float("%.6f" % v) for v in row] for row in a]).astype(np.float32) for a in (pos, power)]
    return lay, path, as_read[0], as_read[1]


# a mesh of two triangles whose box is 40 x 4 x 40
SCENE = """<?xml version="1.0"?>
<scene><material name="m" shader="phong"><mattr name="diffuse" value="0.5 0.5 0.5"/></material>
<object type="mesh" name="o"><matref name="m"/><mesh>
<vertex id="0" val="-20 0 -20"/><vertex id="1" val="20 4 20"/><vertex id="2" val="-20 0 20"/><vertex id="3" val="20 0 -20"/>
<face><vref vertex="0"/><vref vertex="1"/><vref vertex="2"/></face><face><vref vertex="0"/><vref vertex="3"/><vref vertex="1"/></face>
</mesh></object>
<light type="point" color="1.0"><xform pos="0 8 0"/></light>
<camera type="target" fov="50.0"><xform pos="0 7 16"/><target><xform pos="0 0 0"/></target></camera></scene>
"""


@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("k", [0, 1, 8, 50, 100, 600])
def test_gather_selects_the_k_nearest(gpu_lib, dump, which, k):
    lay, path, pos, power = dump
    frac = np.float32(0.5 / np.sqrt(40.0 ** 2 + 4.0 ** 2 + 40.0 ** 2))
    rad = np.sqrt(40.0 ** 2 + 4.0 ** 2 + 40.0 ** 2) * float(frac) if k == 0 else 0.5
    g = gpu_lib.GpuRenderer(width=64, height=64, caust_k=k, gi_k=k, gather_rcap=0.5, gather_dist=float(frac), caust_photons=1000,
                            gi_photons=1000)
    g.load_xml(SCENE)
    g.build(0, 0)
    assert g.restore_photons(which, path) == len(pos)
    q = np.stack([c for c, _ in lay.values()]).astype(np.float32)
    qd = torch.tensor(q, device="cuda")
    nd = torch.tensor([[0.0, 1.0, 0.0]] * len(q), device="cuda")
    out = torch.empty((len(q), 3), device="cuda")
    g.photon_gather(which, qd, nd, out)
    got = out.cpu().numpy().astype(np.float64)
    g.close()
    for i, name in enumerate(lay):
        want = _expected(pos, power, q[i], k, which, rad)
        if not np.isfinite(want).all():
            assert not np.isfinite(got[i]).any(), name     # every photon at the query: the disc has no area
            continue
        err = np.abs(got[i] - want) / np.maximum(np.abs(want), 1e-9)
        assert (err <= BOUND).all(), (name, got[i], want)


def _spread3(v):
    r = np.zeros_like(v)
    for b in range(10):
        r |= ((v >> b) & 1) << (3 * b)
    return r


@pytest.mark.parametrize("n", [40, 3000, 60000])
@pytest.mark.parametrize("k", [0, 20])
def test_gather_grid(gpu_lib, tmp_path, n, k):
    """Random maps of sizes that take each cell width, photons and queries
    inside, on the border of and outside the scene's box, every query against
    all photons in double; and the order programs read the photons in: Morton
    order of cells twice the radius, ties as given."""
    rng = np.random.default_rng(n + k)
    frac = np.float32(0.5 / np.sqrt(40.0 ** 2 + 4.0 ** 2 + 40.0 ** 2))
    rad = np.sqrt(40.0 ** 2 + 4.0 ** 2 + 40.0 ** 2) * float(frac) if k == 0 else 0.5
    pos = rng.uniform((-20.5, -0.4, -20.5), (20.5, 4.4, 20.5), (n, 3))
    pos[: n // 4] = rng.uniform((-1, 1, -1), (1, 1.2, 1), (n // 4, 3))
    pos[n // 4: n // 3, 0] = rng.choice([-20.0, 20.0], n // 3 - n // 4)
    power = rng.uniform(0.5, 2.0, (n, 3))
    path = str(tmp_path / "photons")
    with open(path, "w") as f:
        f.write("energy 300.0\n")
        for p, c in zip(pos, power):
            f.write("<%.6f %.6f %.6f> <0.0 -1.0 0.0> <0.0 1.0 0.0> <%.6f %.6f %.6f>\n" % (*p, *c))
    pos, power = [np.array([[float("%.6f" % v) for v in row] for row in a]).astype(np.float32) for a in (pos, power)]
    g = gpu_lib.GpuRenderer(width=64, height=64, caust_k=k, gi_k=k, gather_rcap=0.5, gather_dist=float(frac), caust_photons=1000,
                            gi_photons=1000)
    g.load_xml(SCENE)
    g.build(0, 0)
    assert g.restore_photons(1, path) == n
    near = pos[rng.integers(0, n, 300)] + rng.uniform(-0.3, 0.3, (300, 3))
    far = rng.uniform((-21, -1, -21), (21, 5, 21), (100, 3))
    q = np.concatenate([near, far, [[-20, 0, -20], [20, 4, 20], [1000, 0, 0], [0, -1000, 0]]]).astype(np.float32)
    out = torch.empty((len(q), 3), device="cuda")
    g.photon_gather(1, torch.tensor(q, device="cuda"), torch.tensor([[0.0, 1.0, 0.0]] * len(q), device="cuda"), out)
    got = out.cpu().numpy().astype(np.float64)
    want = np.stack([_expected(pos, power, p, k, 1, rad) for p in q])
    assert (want > 0).any()
    assert (np.abs(got - want) <= BOUND * np.maximum(np.abs(want), 1e-9)).all()
    ph = g.photons(1)
    g.close()
    lo = np.float64([-20, 0, -20])
    cell = float(np.float32(2.0 * rad))
    while cell < 2.0 * rad:
        cell = float(np.nextafter(np.float32(cell), np.float32(np.inf)))
    dims = np.floor(np.float64([40, 4, 40]) / (2.0 * rad)).astype(np.int64) + 1
    c = np.clip(np.floor((pos.astype(np.float64) - lo) / cell).astype(np.int64), 0, dims - 1)
    order = np.argsort(_spread3(c[:, 0]) | _spread3(c[:, 1]) << 1 | _spread3(c[:, 2]) << 2, kind="stable")
    assert np.array_equal(ph[:, 0:3], pos[order]) and np.array_equal(ph[:, 9:12], power[order])


@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("k", [0, 1, 8, 50, 100])
def test_gather_of_many_points(gpu_lib, dump, which, k):
    """The same selections asked for 32,768 and more times in one call, where
    a thread answers the queries that see few photons and lists the others:
    every copy of a query gets the same answer."""
    lay, path, pos, power = dump
    frac = np.float32(0.5 / np.sqrt(40.0 ** 2 + 4.0 ** 2 + 40.0 ** 2))
    rad = np.sqrt(40.0 ** 2 + 4.0 ** 2 + 40.0 ** 2) * float(frac) if k == 0 else 0.5
    rng = np.random.default_rng(9)
    q = np.stack([c for c, _ in lay.values()]).astype(np.float32)
    # off the centres too: the edges of the discs, between layouts, outside the box
    q = np.concatenate([q, q + rng.uniform(-0.6, 0.6, q.shape).astype(np.float32), rng.uniform((-21, -1, -21), (21, 5, 21), (40, 3)).astype(np.float32)])
    copies = 32768 // len(q) + 2
    g = gpu_lib.GpuRenderer(width=64, height=64, caust_k=k, gi_k=k, gather_rcap=0.5, gather_dist=float(frac), caust_photons=1000,
                            gi_photons=1000)
    g.load_xml(SCENE)
    g.build(0, 0)
    g.restore_photons(which, path)
    qd = torch.tensor(np.tile(q, (copies, 1)), device="cuda")
    nd = torch.tensor([[0.0, 1.0, 0.0]], device="cuda").repeat(len(qd), 1).contiguous()
    out = torch.full((len(qd), 3), -1.0, device="cuda")
    g.photon_gather(which, qd, nd, out)
    got = out.cpu().numpy().astype(np.float64).reshape(copies, len(q), 3)
    g.close()
    assert np.array_equal(got, np.broadcast_to(got[0], got.shape), equal_nan=True)
    for i in range(len(q)):
        want = _expected(pos, power, q[i], k, which, rad)
        if not np.isfinite(want).all():
            assert not np.isfinite(got[0, i]).any()
            continue
        assert (np.abs(got[0, i] - want) <= BOUND * np.maximum(np.abs(want), 1e-9)).all(), (i, got[0, i], want)
