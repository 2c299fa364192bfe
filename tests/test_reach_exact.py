"""Hits that the objects' own boxes could lose, exactly as the FP32 oracle
finds them: segments that end before the cylinder they report (the reference's
cylinder returns the far root beyond the segment's end where the near one is
behind the origin or beside the cylinder), quadrics whose extent the octree
does not know (an octree of one leaf tests every object, so that nothing but
the object boxes can lose a hit), and rays that graze unit-sized objects from
hundreds of units away.  By a warp per ray and by streams of rays."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HEAD = ('<?xml version="1.0"?>\n<scene>\n<material name="m" shader="phong"><mattr name="diffuse" value="0.5 0.5 0.5"/></material>\n')
TAIL = ('<light type="point" color="1.0"><xform pos="0 12 0"/></light>\n'
        '<camera type="target" fov="50.0"><xform pos="0 7 16"/><target><xform pos="0 0 0"/></target></camera></scene>\n')
TETRA = "<mesh>" + "".join('<vertex id="%d" val="%s"/>' % (i, v) for i, v in enumerate(["0 1 0", "1 -1 1", "-1 -1 1", "0 -1 -1"])) + "".join(
    "<face>%s</face>" % "".join('<vref vertex="%d"/>' % v for v in f) for f in ((0, 1, 2), (0, 2, 3), (0, 3, 1), (1, 3, 2))) + "</mesh>"


def _scene(objects):
    """objects: (kind, transform elements, shape element)"""
    return HEAD + "".join('<object type="%s" name="o%d"><matref name="m"/>%s%s</object>\n' % (k, i, xf, body)
                          for i, (k, xf, body) in enumerate(objects)) + TAIL


def _both(gpu_lib, oracle_lib, xml, o, d, tm, mid, interval, warp_rays, **over):
    """(object, face, distance, tie) of the device and of the oracle"""
    opts = dict(width=64, height=64, mblur=1, shutter=20)
    opts.update(over)
    n = len(o)
    orc = oracle_lib.Oracle(fp64=False, rng_mode=1, **opts)
    orc.load_xml(xml)
    orc.prepare(mid)
    want = orc.cast_rays(o.astype(np.float64), d.astype(np.float64), tm)
    g = gpu_lib.GpuRenderer(**opts)
    g.load_xml(xml)
    g.set_tuning(warp_rays=warp_rays)
    g.build(*interval)
    obj, prim = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    t = torch.empty(n, device="cuda")
    tie = torch.empty(n, dtype=torch.uint8, device="cuda")
    g.cast_rays(torch.tensor(o, device="cuda"), torch.tensor(d, device="cuda"), torch.tensor(tm, device="cuda"), obj, prim, t, tie)
    got = [x.cpu().numpy() for x in (obj, prim, t, tie)]
    g.close()
    return got, want


def _check(got, want):
    ok = ~((got[3] > 0) | (want[3] > 0))          # ties: either face may be reported
    assert ok.mean() > 0.99
    hit = want[0] >= 0
    bad = np.flatnonzero((got[0] != want[0]) & ok)
    assert len(bad) == 0, (len(bad), got[0][bad][:5], want[0][bad][:5], want[2][bad][:5])
    assert (got[1] == want[1])[ok & hit].all()
    assert np.array_equal(got[2][ok & hit], want[2][ok & hit].astype(np.float32))


STILL = '<xform pos="%s"/>'
MOVE = '<xform interpolate="linear" time="0" pos="%s"/><xform time="100" pos="%s"/>'
CYLINDERS = [("cylinder", STILL % "3 0 0", '<cylinder rad="0.5" start="0" end="2"/>'),
             ("cylinder", '<xform pos="-4 1 2" axisrot="50 1 0.3 0.2"/>', '<cylinder rad="0.8" start="-1" end="0.5"/>'),
             ("cylinder", MOVE % ("0 0 -5", "0 1 -4"), '<cylinder rad="0.6" start="-0.5" end="1.5"/>'),
             ("sphere", STILL % "-8 0 0", '<sphere rad="1"/>'), ("sphere", STILL % "3 -1.5 0.2", '<sphere rad="0.3"/>')]


@pytest.mark.parametrize("warp_rays", [16384, 0])
@pytest.mark.parametrize("length", [0.3, 1.5])
def test_segments_that_end_before_a_cylinder(gpu_lib, oracle_lib, warp_rays, length):
    rng = np.random.default_rng(5)
    n = 16000
    at = np.float64([[3, 1, 0], [-4, 1, 2], [0, 1, -4.5]])[np.arange(n) % 3]
    o = (at + rng.uniform(-2.2, 2.2, (n, 3)) * (0.4, 1, 0.4)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True) * length).astype(np.float32)
    # straight up through the first cylinder's open end
    o[0], d[0] = (3, -0.5, 0), (0.1, 0.3, 0)
    tm = rng.integers(30, 51, n).astype(np.int32)
    got, want = _both(gpu_lib, oracle_lib, _scene(CYLINDERS), o, d, tm, 40, (30, 50), warp_rays)
    beyond = (want[0] >= 0) & (want[2] > 1)
    assert want[0][0] == 0 and want[2][0] > 4.9 and beyond.sum() > 200
    _check(got, want)


FORMS = ['<xform pos="%s" scale="2.5 0.4 1.5"/>', '<xform pos="%s" axisrot="50 1 0.3 0.2" scale="1 2 0.7"/>', STILL,
         '<xform interpolate="linear" time="0" pos="%s"/><xform time="30" pos="%s"/><xform time="80" pos="%s"/>',
         '<xform interpolate="linear" extrapolate="repeat" time="10" pos="%s" scale="2 0.5 1"/><xform time="25" pos="%s" scale="2 0.5 1"/>']
SHAPES = {"sphere": '<sphere rad="0.8"/>', "cylinder": '<cylinder rad="0.5" start="-0.5" end="1.5"/>', "mesh": TETRA}


@pytest.mark.parametrize("warp_rays", [16384, 0])
def test_quadrics_beyond_their_bounds(gpu_lib, oracle_lib, warp_rays):
    rng = np.random.default_rng(4)
    objects = []
    for f in FORMS:
        for kind, body in SHAPES.items():
            p = rng.uniform((-9, 0, -9), (9, 5, 9))
            at = tuple("%.3f %.3f %.3f" % tuple(p + s) for s in ((0, 0, 0), (1.5, 0.5, -1), (0.5, 2, 1)))
            objects.append((kind, f % at[:f.count("%s")], body))
    n = 16000
    o = rng.uniform((-12, -2, -12), (12, 8, 12), (n, 3)).astype(np.float32)
    d = (rng.uniform((-9, 0, -9), (9, 5, 9), (n, 3)) - o).astype(np.float32) * 4
    tm = rng.integers(30, 51, n).astype(np.int32)
    got, want = _both(gpu_lib, oracle_lib, _scene(objects), o, d, tm, 40, (30, 50), warp_rays, scnoct_max_items=1000)
    _check(got, want)
    # each object by the device itself
    assert (np.bincount(got[0][got[0] >= 0], minlength=len(objects)) >= 30).all()


@pytest.mark.parametrize("warp_rays", [16384, 0])
@pytest.mark.parametrize("far", [100.0, 1000.0, 8000.0])
def test_grazing_from_afar(gpu_lib, oracle_lib, warp_rays, far):
    rng = np.random.default_rng(int(far))
    objects = [("sphere", STILL % "0 0 0", '<sphere rad="1"/>'), ("mesh", STILL % "4 0 0", TETRA),
               ("sphere", '<xform pos="-4 0 0" axisrot="40 1 2 0" scale="2 0.5 1"/>', '<sphere rad="0.7"/>'),
               ("sphere", MOVE % ("0 4 0", "0 4.5 1"), '<sphere rad="1"/>'), ("mesh", MOVE % ("0 -4 0", "1 -4 0.5"), TETRA),
               ("cylinder", STILL % "0 0 4", '<cylinder rad="0.7" start="-1" end="1"/>')]
    at = np.float64([[0, 0, 0], [4, 0, 0], [-4, 0, 0], [0, 4.2, 0.4], [0.4, -4, 0.2], [0, 0, 4]])
    n = 16000
    away = rng.normal(size=(n, 3))
    away /= np.linalg.norm(away, axis=1, keepdims=True)
    side = np.cross(away, rng.normal(size=(n, 3)))
    side /= np.linalg.norm(side, axis=1, keepdims=True)
    # aimed at the edge: a float or so of the origin's size inside or outside a unit sphere's, else anywhere near it
    miss = np.where(np.arange(n) % 2 == 0, 1 + rng.uniform(-1, 1, n) * far * 2.0 ** -21, rng.uniform(0.3, 1.2, n))
    aim = at[np.arange(n) % 6] + side * miss[:, None]
    o = (aim + away * far).astype(np.float32)
    d = ((aim - o) * 1.5).astype(np.float32)
    tm = rng.integers(30, 51, n).astype(np.int32)
    got, want = _both(gpu_lib, oracle_lib, _scene(objects), o, d, tm, 40, (30, 50), warp_rays, scnoct_max_items=1000)
    assert (np.bincount(want[0][want[0] >= 0], minlength=6) > 200).all()
    _check(got, want)
