"""The lights' projection maps made in groups of few lights and of few pairs
of a light sample and an object, as scenes of very many of either need them,
so that their workspace stays bounded: the same photons as from one group, for
jobs and lights that a group's end splits."""
import numpy as np
import pytest
import torch

from test_projmaps import _cases, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group", [1, 7, 100, 301, 5000])
@pytest.mark.parametrize("name", ["many", "moving", "above", "inside a diffuse box"])
def test_groups_give_the_same_photons(gpu_lib, name, group):
    objects, lights, moving = _cases()[name]
    lights = lights + [("point", "4 6 -3"), ("sphere", "-5 8 2"), ("box", "0 11 4")]
    opts = dict(width=32, height=32, caust_photons=3000, gi_photons=3000, caust_k=8, gi_k=8, iter=4, min_samples=1, max_samples=1)
    if moving:
        opts.update(mblur=1, shutter=20)
    got, batch = [], []
    for size in (0, group):
        g = gpu_lib.GpuRenderer(**opts)
        g.load_xml(_scene(objects, lights, moving))
        g.set_faults(photon_group=size)
        try:
            g.shoot_photons(*((30, 50) if moving else (0, 0)))
            got.append([g.photons(which).copy() for which in (0, 1)])
            jobs = [(40 + 5 * k, torch.zeros((32, 32, 4), device="cuda")) for k in range(3)]
            g.render_batch(jobs)
            batch.append([j[1].cpu().numpy() for j in jobs])
        finally:
            g.set_faults()
        g.close()
    for a, b in zip(*got):
        assert len(a) == len(b) and np.array_equal(a, b)
    for a, b in zip(*batch):
        assert np.abs(a - b).max() <= 1e-5 * np.abs(a).max()


def test_workspace_is_bounded(gpu_lib):
    """8,192 objects seen from 12 sphere lights at both ends of an interval:
    1.6 million pairs, 113 MB in one go, 75 MB in groups."""
    rng = np.random.default_rng(1)
    objects = [(rng.uniform((-30, 0.3, -30), (30, 3, 30)), 0.1, k % 4 == 0) for k in range(8191)]
    lights = [("sphere", "%d %d %d" % (3 * k - 18, 9, k % 5)) for k in range(12)]
    xml = _scene(objects, lights, True)
    g = gpu_lib.GpuRenderer(width=32, height=32, caust_photons=2000, gi_photons=2000, caust_k=8, gi_k=8, iter=3, mblur=1, shutter=20)
    g.load_xml(xml)
    g.build(30, 50)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    g.shoot_photons(30, 50)
    used = free - torch.cuda.mem_get_info()[0]
    g.close()
    assert used < 96 << 20, used
