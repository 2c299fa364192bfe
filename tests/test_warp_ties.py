"""Ties of small calls: a warp per ray (calls of up to 16,384 rays) must report
what the streams of rays do where flat meshes of several objects lie in one
plane, so that a ray meets two of them at one distance, or a float apart, and
the entry distance of a flat box is the hit's own, rounding aside."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

def _mesh(vertices, faces):
    return "<mesh>" + "".join('<vertex id="%d" val="%s"/>' % (i, v) for i, v in enumerate(vertices)) + "".join(
        "<face>%s</face>" % "".join('<vref vertex="%d"/>' % v for v in f) for f in faces) + "</mesh>"


QUAD = _mesh(["-2 0 -2", "2 0 -2", "2 0 2", "-2 0 2"], ((0, 2, 1), (0, 3, 2)))
TETRA = _mesh(["0 1 0", "1 -1 1", "-1 -1 1", "0 -1 -1"], ((0, 1, 2), (0, 2, 3), (0, 3, 1), (1, 3, 2)))


def _xml(seed, n):
    """Quads in planes of integer height (some scaled or turned in their plane,
    some upright) among tetrahedra and spheres, which spread a ray's steps"""
    rng = np.random.default_rng(seed)
    out = ['<?xml version="1.0"?>\n<scene>\n<material name="d" shader="phong"><mattr name="diffuse" value="0.5 0.5 0.4"/></material>\n']
    forms = ["", ' scale="%.3f %.3f %.3f"', ' axisrot="90 0 1 0"', ' axisrot="90 1 0 0"']
    for k in range(n):
        p = rng.integers(-3, 4, 3)
        form = forms[rng.integers(0, 4)]
        if "%" in form:
            form = form % tuple(rng.uniform(0.3, 2, 3))
        kind, body = (("mesh", QUAD), ("mesh", QUAD), ("mesh", TETRA), ("sphere", '<sphere rad="0.4"/>'))[k % 4]
        out.append('<object type="%s" name="q%d"><matref name="d"/><xform pos="%.2f %.2f %.2f"%s/>%s</object>\n' % (kind, k, *p, form, body))
    out.append('<light type="point" color="1.0"><xform pos="0 9 0"/></light>\n'
               '<camera type="target" fov="50.0"><xform pos="0 7 16"/><target><xform pos="0 0 0"/></target></camera></scene>\n')
    return "".join(out)


@pytest.mark.parametrize("seed", [1, 2])
@pytest.mark.parametrize("objects", [40, 120])
@pytest.mark.parametrize("length", [1.0, 9.0])
def test_warps_report_what_streams_do(gpu_lib, objects, length, seed):
    rng = np.random.default_rng(3)
    xml = _xml(seed, objects)
    n = 16000
    o = rng.uniform((-5, -5, -5), (5, 5, 5), (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True) * length).astype(np.float32)
    got = []
    for warp_rays in (16384, 0):
        g = gpu_lib.GpuRenderer(width=32, height=32)
        g.load_xml(xml)
        g.set_tuning(warp_rays=warp_rays)
        g.build(0, 0)
        out = [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2)] + [
            torch.empty(n, device="cuda"), torch.empty(n, dtype=torch.uint8, device="cuda")]
        g.cast_rays(torch.tensor(o, device="cuda"), torch.tensor(d, device="cuda"), None, *out)
        got.append([x.cpu().numpy() for x in out])
        g.close()
    assert got[1][3].sum() > 20
    for a, b in zip(*got):
        assert np.array_equal(a, b), (np.flatnonzero(a != b)[:5], (a != b).sum())
