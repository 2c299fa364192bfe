"""Reading a photon map (get_photons, dumps): the first photons of the whole
map's order for any capacity, with no device memory to allocate -- after a
shot of both maps, of one, and of a map restored from a dump."""
import ctypes

import numpy as np
import pytest

from test_projmaps import _cases, _scene

pytestmark = pytest.mark.gpu


def _read(g, which, cap):
    out = np.full((cap + 1, 16), 7.0, np.float32)
    n = ctypes.c_int()
    g._chk(g.L.sray_gpu_get_photons(which, out.ctypes.data_as(ctypes.c_void_p), cap, ctypes.byref(n)))
    assert (out[min(cap, n.value):] == 7.0).all()
    return out[:min(cap, n.value)], n.value


@pytest.mark.parametrize("counts", [(5000, 20000), (20000, 0), (0, 20000)])
def test_without_memory_to_allocate(gpu_lib, tmp_path, counts):
    objects, lights, moving = _cases()["many"]
    xml = _scene(objects, lights, moving)
    opts = dict(width=32, height=32, caust_photons=counts[0], gi_photons=counts[1], caust_k=8, gi_k=8, iter=4)
    g = gpu_lib.GpuRenderer(**opts)
    g.load_xml(xml)
    g.shoot_photons(0, 0)
    dump = str(tmp_path / "dump")
    for which in (0, 1):
        whole = g.photons(which).copy()
        assert (len(whole) > 0) == (counts[which] > 0)
        g.set_faults(fail_alloc_after=0)
        try:
            for cap in (1, 2, 31, len(whole) // 2 + 1, len(whole), len(whole) + 5):
                if len(whole):
                    part, n = _read(g, which, cap)
                    assert n == len(whole) and np.array_equal(part, whole[:cap])
            g.dump_photons(which, dump + str(which))
        finally:
            g.set_faults()
    g.close()
    # a context that has shot nothing holds no buffers but the map's
    for which in (0, 1):
        if not counts[which]:
            continue
        g = gpu_lib.GpuRenderer(**opts)
        g.load_xml(xml)
        g.build(0, 0)
        n = g.restore_photons(which, dump + str(which))
        g.set_faults(fail_alloc_after=0)
        try:
            small, _ = _read(g, which, 100)
            held, _ = _read(g, which, n)
            g.dump_photons(which, dump + "again")
        finally:
            g.set_faults()
        whole = g.photons(which)
        g.close()
        assert np.array_equal(held, whole) and np.array_equal(small, whole[:100])
        assert sorted(open(dump + "again")) == sorted(open(dump + str(which)))
