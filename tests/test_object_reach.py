"""Hits of objects whose own extent differs from the bounds the scene octree
lists them by: scaled spheres (the reference's bounds ignore the scaling, so
the octree lists them in too few leaves, and what it lists decides), rotated
and scaled cylinders, meshes and spheres moving on linear, step and repeated
keys, rotating and cubic tracks (whose extent is not known), at times over
the frame's whole table -- against the FP32 oracle, bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _scene():
    mat = '<material name="m" shader="phong"><mattr name="diffuse" value="0.5 0.5 0.5"/></material>\n'
    tetra = "".join('<vertex id="%d" val="%s"/>' % (i, v) for i, v in enumerate(["0 1 0", "1 -1 1", "-1 -1 1", "0 -1 -1"]))
    tetra += "".join("<face>%s</face>" % "".join('<vref vertex="%d"/>' % v for v in f) for f in ((0, 1, 2), (0, 2, 3), (0, 3, 1), (1, 3, 2)))
    body = {"s": '<sphere rad="0.8"/>', "c": '<cylinder rad="0.5" start="-0.5" end="1.5"/>', "m": "<mesh>%s</mesh>" % tetra}
    kind = {"s": "sphere", "c": "cylinder", "m": "mesh"}
    forms = ['<xform pos="%s" scale="2.5 0.4 1.5"/>', '<xform pos="%s" axisrot="50 1 0.3 0.2" scale="1 2 0.7"/>', '<xform pos="%s"/>',
             '<xform interpolate="linear" time="0" pos="%s"/><xform time="30" pos="%s"/><xform time="80" pos="%s"/>',
             '<xform interpolate="step" time="0" pos="%s"/><xform time="35" pos="%s"/>',
             '<xform interpolate="linear" extrapolate="repeat" time="10" pos="%s"/><xform time="25" pos="%s"/>',
             '<xform interpolate="linear" time="0" pos="%s" axisrot="0 0 1 0"/><xform time="60" pos="%s" axisrot="90 0 1 0"/>',
             '<xform interpolate="cubic" time="0" pos="%s"/><xform time="25" pos="%s"/><xform time="60" pos="%s"/>']
    rng = np.random.default_rng(4)
    out, k = [], 0
    for f in forms:
        for b in body:
            p = rng.uniform((-9, 0, -9), (9, 5, 9))
            at = tuple("%.3f %.3f %.3f" % tuple(p + d) for d in ((0, 0, 0), (1.5, 0.5, -1), (0.5, 2, 1)))
            out.append('<object type="%s" name="o%d"><matref name="m"/>%s%s</object>\n' % (kind[b], k, f % at[:f.count("%s")], body[b]))
            k += 1
    return ('<?xml version="1.0"?>\n<scene>\n' + mat + "".join(out) + '<light type="point" color="1.0"><xform pos="0 12 0"/></light>\n'
            '<camera type="target" fov="50.0"><xform pos="0 7 16"/><target><xform pos="0 0 0"/></target></camera></scene>\n')


@pytest.mark.parametrize("n", [4000, 40000])       # a warp per ray; streams of rays
@pytest.mark.parametrize("depth,items", [(8, 2), (3, 8)])
def test_hits_within_reach(gpu_lib, oracle_lib, n, depth, items):
    xml = _scene()
    opts = dict(width=64, height=64, mblur=1, shutter=20, scnoct_max_depth=depth, scnoct_max_items=items)
    rng = np.random.default_rng(n)
    o = rng.uniform((-12, -2, -12), (12, 8, 12), (n, 3)).astype(np.float32)
    d = (rng.uniform((-9, 0, -9), (9, 5, 9), (n, 3)) - o).astype(np.float32) * 4
    tm = rng.integers(30, 51, n).astype(np.int32)
    orc = oracle_lib.Oracle(fp64=False, rng_mode=1, **opts)
    orc.load_xml(xml)
    orc.prepare(40)
    want = orc.cast_rays(o.astype(np.float64), d.astype(np.float64), tm)
    g = gpu_lib.GpuRenderer(**opts)
    g.load_xml(xml)
    g.build(30, 50)
    obj, prim = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    t = torch.empty(n, device="cuda")
    tie = torch.empty(n, dtype=torch.uint8, device="cuda")
    g.cast_rays(torch.tensor(o, device="cuda"), torch.tensor(d, device="cuda"), torch.tensor(tm, device="cuda"), obj, prim, t, tie)
    got = [x.cpu().numpy() for x in (obj, prim, t, tie)]
    g.close()
    ok = ~((got[3] > 0) | (want[3] > 0))
    hit = want[0] >= 0
    assert hit.mean() > 0.1 and len(np.unique(want[0])) >= 20
    # the scaled quadrics (objects 0, 1, 3, 4) reach beyond the leaves that list
    # them: a hit outside may lie before the leaf, where the oracle, which visits
    # every leaf of the ray, counts it and the device octree, which stops at the
    # closest hit so far, may not; such a ray reports the oracle's hit or a later one
    beyond = hit & np.isin(want[0], (0, 1, 3, 4))
    assert ((got[0] == want[0]) | (got[0] < 0) | (got[2] >= want[2].astype(np.float32)))[beyond].all()
    ok &= ~beyond
    assert (got[0] == want[0])[ok].all()
    assert (got[1] == want[1])[ok & hit].all()
    assert np.array_equal(got[2][ok & hit], want[2][ok & hit].astype(np.float32))
