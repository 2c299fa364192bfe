"""The cell of a projection map that holds an object's centre, at directions
where a cell ends: lights at 45 degrees' elevation or azimuth to small objects,
where the last bit of the angle decides the cell.  The objects are too small
for a corner of a cell to see them, so that this cell is all they set: both
photon maps equal to the FP32 oracle's, photon for photon."""
import itertools

import numpy as np
import pytest

from test_projmaps import _scene

pytestmark = pytest.mark.gpu

RAD = 0.25
LIGHT = (0.0, 40.0, 0.0)
OFF = (0.1, 40.0, 0.2)      # differences to it are rounded


def _signed(x, y, z):
    return [(a * x, b * y, c * z) for a, b, c in itertools.product((-1, 1), repeat=3)]


# y^2 = x^2 + z^2: the edge of rows 8 and 24
TRIPLES = [(15, 17, 8), (8, 17, 15), (12, 13, 5), (5, 13, 12), (16, 20, 12), (24, 25, 7), (20, 29, 21), (21, 29, 20)]
DIRS = {"elevation %d %d %d" % t: (LIGHT, _signed(*t)) for t in TRIPLES}
DIRS["level"] = (LIGHT, [(x, 0, z) for x, z in ((9, 4), (-9, 4), (7, -10), (-5, -11))])
DIRS["azimuth"] = (LIGHT, [(sx * d, y, sz * d) for d in (7, 11, 13) for y in (3, -4) for sx, sz in itertools.product((-1, 1), repeat=2)]
                   + [(9, 3, 0), (-9, 3, 0), (0, 4, 11), (0, 4, -11)])
DIRS["azimuth, rounded"] = (OFF, [(s * k, 3, s * k) for k in range(7, 14) for s in (-1, 1)] + [(9, 3, 0), (-9, 3, 0), (0, 3, -9), (0, -3, 9)])


@pytest.mark.parametrize("name", sorted(DIRS))
def test_photons_at_cell_ends(gpu_lib, oracle_lib, name):
    light, dirs = DIRS[name]
    stored = 0
    for v in dirs:
        xml = _scene([(tuple(np.add(light, v)), RAD, True)], [("point", "%.1f %.1f %.1f" % light)], False)
        opts = dict(width=32, height=32, caust_photons=800, gi_photons=200, caust_k=8, gi_k=8, iter=5)
        g = gpu_lib.GpuRenderer(**opts)
        g.load_xml(xml)
        o = oracle_lib.Oracle(fp64=False, rng_mode=1, **opts)
        o.load_xml(xml)
        o.prepare(0)
        g.shoot_photons(0, 0)
        for which in (0, 1):
            a, b = g.photons(which)[:, :12], o.photons(which)[:, :12]
            assert len(a) == len(b), (v, which)
            assert np.array_equal(a[np.lexsort(a.T[::-1])], b[np.lexsort(b.T[::-1])]), (v, which)
            stored += len(a)
        g.close()
    assert stored > 0


@pytest.mark.parametrize("light", ["point", "sphere", "box"])
def test_light_at_a_flat_objects_centre(gpu_lib, oracle_lib, light):
    """The direction from the light to the floor's centre has no length, so
    its angles are no numbers (the floor's box is flat: the light is not inside)."""
    xml = _scene([((3, 1.5, 2), 0.7, True)], [(light, "0 0 0")], False).replace("-0.5 -0.25 -1", "0 0 0").replace("0.5 0.25 1", "0 0 0")
    xml = xml.replace('<sphere rad="0.6"/>', '<sphere rad="0"/>')
    opts = dict(width=32, height=32, caust_photons=3000, gi_photons=3000, caust_k=8, gi_k=8, iter=5)
    g = gpu_lib.GpuRenderer(**opts)
    g.load_xml(xml)
    o = oracle_lib.Oracle(fp64=False, rng_mode=1, **opts)
    o.load_xml(xml)
    o.prepare(0)
    g.shoot_photons(0, 0)
    for which in (0, 1):
        a, b = g.photons(which)[:, :12], o.photons(which)[:, :12]
        assert len(a) == len(b) > 0
        assert np.array_equal(a[np.lexsort(a.T[::-1])], b[np.lexsort(b.T[::-1])])
    g.close()
