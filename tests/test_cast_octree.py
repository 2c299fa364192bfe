"""Rays that the octrees must decide, in calls of every route -- a warp per
ray, blocks that follow the octrees themselves, blocks that mark such rays for
a second launch (more than a ray per lane of the GPU) -- and without device
memory to allocate."""
import numpy as np
import pytest
import torch

from sray_gb300 import scenegen

pytestmark = pytest.mark.gpu

LANES = 152 * 8 * 128


def _tied():
    quad = ('<object type="mesh" name="%s"><matref name="d"/><mesh>'
            + "".join('<vertex id="%d" val="%s"/>' % (i, v) for i, v in enumerate(["-20 0 -20", "20 0 -20", "20 0 20", "-20 0 20"]))
            + '<face><vref vertex="0"/><vref vertex="2"/><vref vertex="1"/></face>'
              '<face><vref vertex="0"/><vref vertex="3"/><vref vertex="2"/></face></mesh></object>\n')
    return ('<?xml version="1.0"?>\n<scene>\n<material name="d" shader="phong"><mattr name="diffuse" value="0.5 0.5 0.4"/></material>\n'
            + quad % "a" + quad % "b" + '<object type="sphere" name="c"><matref name="d"/><sphere rad="3"/></object>\n'
            '<light type="point" color="1.0"><xform pos="0 9 0"/></light>\n'
            '<camera type="target" fov="50.0"><xform pos="0 7 16"/><target><xform pos="0 0 0"/></target></camera></scene>\n')


def _outputs(n):
    return [torch.full((n,), 7, dtype=torch.int32, device="cuda") for _ in range(2)] + [
        torch.full((n,), 7.0, device="cuda"), torch.full((n,), 7, dtype=torch.uint8, device="cuda")]


@pytest.mark.parametrize("n", [4096, 4097, LANES, LANES + 1, 3 * LANES + 517])
def test_call_equals_its_pieces(gpu_lib, n):
    rng = np.random.default_rng(n)
    o = torch.tensor(rng.uniform((-22, -4, -22), (22, 9, 22), (n, 3)).astype(np.float32), device="cuda")
    d = torch.tensor((rng.normal(size=(n, 3)) * (1, 0.3, 1) - (0, 1, 0)).astype(np.float32) * 60.0, device="cuda")
    g = gpu_lib.GpuRenderer(width=32, height=32)
    g.load_xml(_tied())
    g.build(0, 0)
    whole, pieces = _outputs(n), _outputs(n)
    g.cast_rays(o, d, None, *whole)
    for a in range(0, n, 4000):        # by warps
        g.cast_rays(o[a:a + 4000].contiguous(), d[a:a + 4000].contiguous(), None, *[p[a:a + 4000] for p in pieces])
    g.close()
    assert 0.2 < whole[3].float().mean() < 0.9 and (whole[0] == 2).any() and (whole[0] == -1).any()
    for a, b in zip(whole, pieces):
        assert torch.equal(a, b)


@pytest.mark.parametrize("n", [16385, 300000])
def test_no_memory_to_allocate(gpu_lib, n):
    rng = np.random.default_rng(n)
    o = torch.tensor(rng.uniform((-40, 0.1, -20), (40, 9, 20), (n, 3)).astype(np.float32), device="cuda")
    d = torch.tensor(rng.normal(size=(n, 3)).astype(np.float32) * 60.0, device="cuda")
    g = gpu_lib.GpuRenderer(**scenegen.scene_opts("production", width=64, height=64))
    g.load(scenegen.write_scene("production", grid=(60, 30), n_inst=12))
    g.build(0, 0)
    first, ref, out = _outputs(1), _outputs(n), _outputs(n)
    g.cast_rays(o[:1].contiguous(), d[:1].contiguous(), None, *first)      # the context's counters
    g.set_faults(fail_alloc_after=0)
    try:
        g.cast_rays(o, d, None, *out)
    finally:
        g.set_faults()
    g.cast_rays(o, d, None, *ref)
    g.close()
    assert (out[0] >= 0).any()
    for a, b in zip(out, ref):
        assert torch.equal(a, b)
