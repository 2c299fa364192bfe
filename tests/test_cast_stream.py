"""Closest hits of a program's own rays, by each of the traversals that a call
of its size takes -- one warp per ray up to 16,384 rays, above that blocks of
128 threads that take their chunk's rays as lanes fall idle -- against the
FP32 oracle: object and face ids and the distance bit for bit, ties as the
octrees report them.  Sizes: a lone ray, the edges of a warp and of a block,
both sides of the rule, a last chunk of few rays, chunks of several rays per
lane."""
import numpy as np
import pytest
import torch

from sray_gb300 import scenegen

pytestmark = pytest.mark.gpu

N = 200003


@pytest.fixture(scope="module", params=["terrain", "movers"])
def cast_pair(request, gpu_lib, oracle_lib):
    if request.param == "terrain":
        path, t1 = scenegen.write_scene("production", grid=(60, 30), n_inst=12), 0
        opts = scenegen.scene_opts("production", width=64, height=64)
        ext = (45.0, 22.0)
    else:
        path, t1 = scenegen.write_scene("batch", seed=1000, tris=12000), 8
        opts = scenegen.scene_opts("production", width=64, height=64, mblur=1, shutter=8)
        ext = (35.0, 17.0)
    rng = np.random.default_rng(3)
    o = rng.uniform((-ext[0], -1.0, -ext[1]), (ext[0], 12.0, ext[1]), (N, 3)).astype(np.float32)
    d = rng.normal(size=(N, 3)).astype(np.float32) * 60.0
    tm = rng.integers(0, t1 + 1, N).astype(np.int32)
    orc = oracle_lib.Oracle(fp64=False, rng_mode=1, **opts)
    orc.load(path)
    orc.prepare(t1 // 2)          # the frame's interval is [0, t1]
    want = orc.cast_rays(o.astype(np.float64), d.astype(np.float64), tm)
    return path, opts, t1, o, d, tm, want


@pytest.mark.parametrize("warp_rays", [16384, 0])
@pytest.mark.parametrize("n", [1, 33, 127, 129, 16384, 16385, 70001, N])
def test_cast_rays_by_size(gpu_lib, cast_pair, n, warp_rays):
    path, opts, t1, o, d, tm, want = cast_pair
    g = gpu_lib.GpuRenderer(**opts)
    g.load(path)
    g.set_tuning(warp_rays=warp_rays)
    g.build(0, t1)
    obj, prim = (torch.full((n,), 7, dtype=torch.int32, device="cuda") for _ in range(2))
    t = torch.full((n,), 7.0, device="cuda")
    tie = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
    times = torch.tensor(tm[:n], device="cuda") if t1 else None
    g.cast_rays(torch.tensor(o[:n], device="cuda"), torch.tensor(d[:n], device="cuda"), times, obj, prim, t, tie)
    got = [x.cpu().numpy() for x in (obj, prim, t, tie)]
    g.close()
    hit = want[0][:n] >= 0
    ok = ~((got[3] > 0) | (want[3][:n] > 0))      # ties: either face may be reported
    assert (got[0] == want[0][:n])[ok].all()
    assert (got[1] == want[1][:n])[ok & hit].all()
    assert np.array_equal(got[2][ok & hit], want[2][:n][ok & hit].astype(np.float32))
    assert (got[1][~hit] == -1).all() and (got[2][~hit] == 0).all()
    if n == N:
        assert hit.any() and (~hit).any()


@pytest.mark.parametrize("n", [1, 64, 5000, 16384])
def test_octree_decided_rays(gpu_lib, n):
    """Two coincident meshes: every hit is a tie that the octrees decide, by the
    ray's own warp in a small call, by a second launch in a large one."""
    quad = ('<object type="mesh" name="%s"><matref name="d"/><mesh>'
            + "".join('<vertex id="%d" val="%s"/>' % (i, v) for i, v in enumerate(["-20 0 -20", "20 0 -20", "20 0 20", "-20 0 20"]))
            + '<face><vref vertex="0"/><vref vertex="2"/><vref vertex="1"/></face>'
              '<face><vref vertex="0"/><vref vertex="3"/><vref vertex="2"/></face></mesh></object>\n')
    xml = ('<?xml version="1.0"?>\n<scene>\n<material name="d" shader="phong"><mattr name="diffuse" value="0.5 0.5 0.4"/></material>\n'
           + quad % "a" + quad % "b" + '<light type="point" color="1.0"><xform pos="0 9 0"/></light>\n'
           '<camera type="target" fov="50.0"><xform pos="0 7 16"/><target><xform pos="0 0 0"/></target></camera></scene>\n')
    rng = np.random.default_rng(n)
    o = torch.tensor(rng.uniform((-15, 2, -15), (15, 9, 15), (n, 3)).astype(np.float32), device="cuda")
    d = torch.tensor((rng.normal(size=(n, 3)) * (1, 0.3, 1) - (0, 1, 0)).astype(np.float32) * 60.0, device="cuda")
    got = []
    for warp_rays in (16384, 0):
        g = gpu_lib.GpuRenderer(width=32, height=32)
        g.load_xml(xml)
        g.set_tuning(warp_rays=warp_rays)
        g.build(0, 0)
        out = [torch.full((n,), 7, dtype=torch.int32, device="cuda") for _ in range(2)]
        out += [torch.full((n,), 7.0, device="cuda"), torch.full((n,), 7, dtype=torch.uint8, device="cuda")]
        g.cast_rays(o, d, None, *out)
        got.append([x.cpu().numpy() for x in out])
        g.close()
    assert (got[0][0] >= 0).any() or n == 1
    for a, b in zip(*got):
        assert np.array_equal(a, b)
