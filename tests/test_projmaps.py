"""The lights' projection maps, seen through the photons they let out: both
photon maps equal to the FP32 oracle's, photon for photon (a photon's power
carries its map's coverage, its direction the map's cells), for lights that
see the objects in the ways the maps distinguish -- inside an object's box,
straight above one, tiny and distant ones, hundreds of them, a light of each
kind, no specular object, an interval with two ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIGHTS = {"point": '<light type="point" color="1.0"><xform pos="%s"/></light>\n',
          "sphere": '<light type="sphere" color="0.8"><xform pos="%s"/><sphere rad="0.6"/></light>\n',
          "box": '<light type="box" color="0.7"><xform pos="%s"/><aabox min="-0.5 -0.25 -1" max="0.5 0.25 1"/></light>\n'}


def _scene(objects, lights, moving):
    out = ['<?xml version="1.0"?>\n<scene>\n<material name="d" shader="phong"><mattr name="diffuse" value="0.5 0.5 0.4"/></material>\n'
           '<material name="g" shader="phong"><mattr name="diffuse" value="0.1 0.1 0.1"/><mattr name="specular" value="0.9 0.9 0.9"/>'
           '<mattr name="refract" value="0.9"/><mattr name="ior" value="1.4"/></material>\n']
    out.append('<object type="mesh" name="f"><matref name="d"/><mesh>%s<face><vref vertex="0"/><vref vertex="2"/><vref vertex="1"/></face>'
               '<face><vref vertex="0"/><vref vertex="3"/><vref vertex="2"/></face></mesh></object>\n'
               % "".join('<vertex id="%d" val="%s"/>' % (i, v) for i, v in enumerate(["-20 0 -20", "20 0 -20", "20 0 20", "-20 0 20"])))
    for k, (p, r, glass) in enumerate(objects):
        xf = '<xform pos="%.4f %.4f %.4f"/>' % tuple(p)
        if moving:
            xf = '<xform interpolate="linear" time="0" pos="%.4f %.4f %.4f"/><xform time="100" pos="%.4f %.4f %.4f"/>' % (*p, *(np.add(p, (3, 1, 2))))
        out.append('<object type="sphere" name="s%d"><matref name="%s"/>%s<sphere rad="%.5f"/></object>\n' % (k, "g" if glass else "d", xf, r))
    for kind, pos in lights:
        out.append(LIGHTS[kind] % pos)
    out.append('<camera type="target" fov="50.0"><xform pos="0 7 16"/><target><xform pos="0 0 0"/></target></camera></scene>\n')
    return "".join(out)


def _cases():
    rng = np.random.default_rng(6)
    some = [((-3, 1, 0), 1.0, True), ((3, 1.5, 2), 0.7, False), ((0, 4, -4), 0.5, True)]
    many = [(rng.uniform((-15, 0.3, -15), (15, 3, 15)), rng.uniform(0.1, 0.5), i % 3 == 0) for i in range(300)]
    tiny = [(rng.uniform((-15, 0.3, -15), (15, 12, 15)), 0.003, True) for i in range(20)]
    return {"inside a box": (some + [((0, 9, 0), 3.0, True)], [("point", "0 9 0")], False),
            "inside a diffuse box": (some + [((0, 9, 0), 3.0, False)], [("sphere", "0 9.5 0")], False),
            "above": ([((0, 1, 0), 1.0, True)], [("point", "0 8 0"), ("box", "0 6 0")], False),
            "no specular": ([((0, 1, 0), 1.0, False)], [("point", "2 8 0")], False),
            "many": (many, [("sphere", "0 9 0"), ("sphere", "-6 7 3"), ("point", "5 8 5")], False),
            "tiny": (tiny, [("box", "1 14 0"), ("point", "0 6 0")], False),
            "moving": (some, [("sphere", "1 8 0"), ("box", "-4 7 1")], True),
            "far": (some, [("point", "900 3000 -700")], False)}


@pytest.mark.parametrize("name", sorted(_cases()))
def test_photons_of_projection_maps(gpu_lib, oracle_lib, name):
    objects, lights, moving = _cases()[name]
    xml = _scene(objects, lights, moving)
    opts = dict(width=32, height=32, caust_photons=3000, gi_photons=3000, caust_k=8, gi_k=8, iter=5)
    if moving:
        opts.update(mblur=1, shutter=20)
    g = gpu_lib.GpuRenderer(**opts)
    g.load_xml(xml)
    o = oracle_lib.Oracle(fp64=False, rng_mode=1, **opts)
    o.load_xml(xml)
    o.prepare(40 if moving else 0)
    t = (30, 50) if moving else (0, 0)
    g.shoot_photons(*t)
    stored = 0
    for which in (0, 1):
        a, b = g.photons(which)[:, :12], o.photons(which)[:, :12]
        assert len(a) == len(b)
        assert np.array_equal(a[np.lexsort(a.T[::-1])], b[np.lexsort(b.T[::-1])])
        stored += len(a)
    g.close()
    assert stored > 0


@pytest.mark.parametrize("n", [1, 31, 5000, 20001, 60000, 320000])
def test_emission_by_count(gpu_lib, oracle_lib, n):
    """The emission gives a photon a lane of its own, or several, by the number
    of photons (2 to 32 photons per warp): the same photons at every count."""
    objects, lights, moving = _cases()["many"]
    xml = _scene(objects, lights, moving)
    opts = dict(width=32, height=32, caust_photons=n, gi_photons=max(1, n // 4), caust_k=8, gi_k=8, iter=4)
    g = gpu_lib.GpuRenderer(**opts)
    g.load_xml(xml)
    o = oracle_lib.Oracle(fp64=False, rng_mode=1, **opts)
    o.load_xml(xml)
    o.prepare(0)
    g.shoot_photons(0, 0)
    for which in (0, 1):
        a, b = g.photons(which)[:, :12], o.photons(which)[:, :12]
        assert len(a) == len(b)
        assert np.array_equal(a[np.lexsort(a.T[::-1])], b[np.lexsort(b.T[::-1])])
    g.close()
