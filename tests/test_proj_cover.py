"""The ordered sum of a projection map's coverage, which one map in some
30,000 needs, for every map (the injected photon groups ask for it): both
photon maps equal to the FP32 oracle's, photon for photon, whose powers carry
the coverages."""
import numpy as np
import pytest

from test_projmaps import _cases, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", sorted(_cases()))
def test_photons_of_ordered_coverages(gpu_lib, oracle_lib, name):
    objects, lights, moving = _cases()[name]
    xml = _scene(objects, lights, moving)
    opts = dict(width=32, height=32, caust_photons=2000, gi_photons=2000, caust_k=8, gi_k=8, iter=5)
    if moving:
        opts.update(mblur=1, shutter=20)
    g = gpu_lib.GpuRenderer(**opts)
    g.load_xml(xml)
    o = oracle_lib.Oracle(fp64=False, rng_mode=1, **opts)
    o.load_xml(xml)
    o.prepare(40 if moving else 0)
    g.set_faults(photon_group=1 << 20)
    try:
        g.shoot_photons(*((30, 50) if moving else (0, 0)))
    finally:
        g.set_faults()
    stored = 0
    for which in (0, 1):
        a, b = g.photons(which)[:, :12], o.photons(which)[:, :12]
        assert len(a) == len(b)
        assert np.array_equal(a[np.lexsort(a.T[::-1])], b[np.lexsort(b.T[::-1])])
        stored += len(a)
    g.close()
    assert stored > 0
