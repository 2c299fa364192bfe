"""The objects' own boxes on the CPU (no GPU): tests/reach_check.cc over the
scene of tests/test_object_reach.py, whose objects have every form of
transform."""
import os
import subprocess

import pytest

from test_object_reach import _scene

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("reach")
    csrc = os.path.join(ROOT, "sray_gb300", "csrc")
    exe = d / "reach_check"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + os.path.join(ROOT, "include"), "-I" + csrc,
                           "-I/usr/local/cuda/include", os.path.join(ROOT, "tests", "reach_check.cc"),
                           os.path.join(csrc, "scene_host.cc"), os.path.join(csrc, "bvh_host.cc"), "-o", str(exe), "-lpthread"])
    path = d / "scene.xml"
    path.write_text(_scene())
    return str(exe), str(path)


@pytest.mark.parametrize("t0,t1,shutter", [(30, 50, 20), (0, 0, 0), (5, 30, 8), (80, 100, 40)])
def test_reach_holds_every_point(check, t0, t1, shutter):
    out = subprocess.run(list(check) + [str(t0), str(t1), str(shutter)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
