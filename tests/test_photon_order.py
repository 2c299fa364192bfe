"""A large emission pass is traced in an order of its own: both photon maps
equal to the FP32 oracle's, photon for photon, on both sides of the size from
which it is (2^20 photons of both maps), with thread- and warp-per-ray passes,
and a second shoot after the first."""
import numpy as np
import pytest

from test_projmaps import _cases, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,ng,warp_rays", [(800000, 248000, 16384), (800000, 250000, 16384), (800001, 250007, 1 << 24)])
def test_photons_of_large_passes(gpu_lib, oracle_lib, nc, ng, warp_rays):
    objects, lights, moving = _cases()["many"]
    xml = _scene(objects, lights, moving)
    opts = dict(width=32, height=32, caust_photons=nc, gi_photons=ng, caust_k=8, gi_k=8, iter=4)
    g = gpu_lib.GpuRenderer(**opts)
    g.load_xml(xml)
    g.set_tuning(warp_rays=warp_rays)
    o = oracle_lib.Oracle(fp64=False, rng_mode=1, **opts)
    o.load_xml(xml)
    o.prepare(0)
    for shoot in range(2):
        g.shoot_photons(0, 0)
        for which in (0, 1):
            a, b = g.photons(which)[:, :12], o.photons(which)[:, :12]
            assert len(a) == len(b)
            assert np.array_equal(a[np.lexsort(a.T[::-1])], b[np.lexsort(b.T[::-1])])
    g.close()
