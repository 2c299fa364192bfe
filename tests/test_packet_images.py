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
