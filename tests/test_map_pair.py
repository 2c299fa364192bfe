"""A frame's two photon maps are built together (one sort, the maps' cells one
after the other).  Each must be the map it is when the other has no photons:
the same photons in the same order and the same estimates, exactly -- with
one map empty, tiny, or ending within, at and past a tile of the sort, and
with grids of different sizes (range gathers against the nearest 8)."""
import numpy as np
import pytest
import torch

from test_projmaps import _cases, _scene

pytestmark = pytest.mark.gpu


def _maps(gpu_lib, xml, pts, nc, ng, ck):
    g = gpu_lib.GpuRenderer(width=32, height=32, caust_photons=nc, gi_photons=ng, caust_k=ck, gi_k=8, iter=4)
    g.load_xml(xml)
    counts = g.shoot_photons(0, 0)
    got = []
    for which in (0, 1):
        out = torch.full((len(pts), 3), 7.0, device="cuda")
        if counts[which]:
            g.photon_gather(which, pts, torch.tensor([[0.0, 1.0, 0.0]], device="cuda").repeat(len(pts), 1), out)
        got.append((g.photons(which).copy(), out.cpu().numpy()))
    g.close()
    return counts, got


@pytest.mark.parametrize("nc,ng,ck", [(1, 1, 8), (5000, 1, 8), (1, 5000, 8), (5000, 0, 8), (0, 5000, 0), (4096, 4096, 0), (30000, 700, 0), (900, 60000, 8), (60000, 60000, 0)])
def test_maps_together_and_alone(gpu_lib, nc, ng, ck):
    objects, lights, moving = _cases()["many"]
    xml = _scene(objects, lights, moving)
    rng = np.random.default_rng(nc + ng)
    pts = torch.tensor(rng.uniform((-15, 0, -15), (15, 0.02, 15), (3000, 3)).astype(np.float32), device="cuda")
    counts, both = _maps(gpu_lib, xml, pts, nc, ng, ck)
    for which, (a, b) in enumerate([(nc, 0), (0, ng)]):
        if not counts[which]:
            continue
        alone, one = _maps(gpu_lib, xml, pts, a, b, ck)
        assert alone[which] == counts[which] and alone[1 - which] == 0
        assert np.array_equal(one[which][0], both[which][0])
        assert np.array_equal(one[which][1], both[which][1])
