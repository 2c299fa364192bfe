"""Primary hits on both sides of the image size from which camera rays are
traced as warp packets (400,000 pixels), at sizes that leave packets of few
pixels at the edges -- against the FP32 oracle, bit for bit."""
import numpy as np
import pytest
import torch

from sray_gb300 import scenegen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(799, 500), (800, 500), (803, 501), (1603, 251)])
@pytest.mark.parametrize("scene", ["small", "terrain"])
def test_primary_hits_by_image_size(gpu_lib, oracle_lib, size, scene):
    w, h = size
    path = scenegen.write_scene("small") if scene == "small" else scenegen.write_scene("production", grid=(60, 30), n_inst=12)
    opts = scenegen.scene_opts("small" if scene == "small" else "production", width=w, height=h)
    g = gpu_lib.GpuRenderer(**opts)
    g.load(path)
    n = w * h
    obj, prim = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    t = torch.empty(n, device="cuda")
    tie = torch.empty(n, dtype=torch.uint8, device="cuda")
    g.primary_hits(obj, prim, t, tie)
    got = [x.cpu().numpy() for x in (obj, prim, t, tie)]
    g.close()
    o = oracle_lib.Oracle(fp64=False, rng_mode=1, **opts)
    o.load(path)
    want = o.primary_hits()
    ok = ~((got[3] > 0) | (want[3] > 0))
    hit = want[0] >= 0
    assert hit.any()
    assert (got[0] == want[0])[ok].all() and (got[1] == want[1])[ok & hit].all()
    assert np.array_equal(got[2][ok & hit], want[2][ok & hit].astype(np.float32))


@pytest.mark.parametrize("size", [(800, 500), (803, 501), (1603, 251)])
@pytest.mark.parametrize("scene", ["ties", "movers"])
def test_primary_hits_of_packets_and_single_rays(gpu_lib, size, scene):
    """Images large enough for packets, by packets and by a warp per ray (a
    tuning that no image passes): every output the same, where the octrees
    decide each hit (two coincident meshes) and with moving spheres."""
    w, h = size
    quad = ('<object type="mesh" name="%s"><matref name="d"/><mesh>'
            + "".join('<vertex id="%d" val="%s"/>' % (i, v) for i, v in enumerate(["-20 0 -20", "20 0 -20", "20 0 20", "-20 0 20"]))
            + '<face><vref vertex="0"/><vref vertex="2"/><vref vertex="1"/></face>'
              '<face><vref vertex="0"/><vref vertex="3"/><vref vertex="2"/></face></mesh></object>\n')
    xml = ('<?xml version="1.0"?>\n<scene>\n<material name="d" shader="phong"><mattr name="diffuse" value="0.5 0.5 0.4"/></material>\n'
           + quad % "a" + quad % "b" + '<light type="point" color="1.0"><xform pos="0 9 0"/></light>\n'
           '<camera type="target" fov="50.0"><xform pos="0 7 16"/><target><xform pos="0 0 0"/></target></camera></scene>\n')
    got = []
    for warp_rays in (0, 1 << 24):
        if scene == "ties":
            g = gpu_lib.GpuRenderer(width=w, height=h)
            g.load_xml(xml)
        else:
            g = gpu_lib.GpuRenderer(**scenegen.scene_opts("production", width=w, height=h, mblur=1, shutter=8))
            g.load(scenegen.write_scene("batch", seed=1000, tris=12000))
        g.set_tuning(warp_rays=warp_rays)
        n = w * h
        out = [torch.full((n,), 7, dtype=torch.int32, device="cuda") for _ in range(2)]
        out += [torch.full((n,), 7.0, device="cuda"), torch.full((n,), 7, dtype=torch.uint8, device="cuda")]
        g.primary_hits(*out, msec=40 if scene == "movers" else 0)
        got.append([x.cpu().numpy() for x in out])
        g.close()
    assert (got[0][0] >= 0).any()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
