"""A program that resets the device (which ends its own context on it) and goes on: contexts
and guides made after it have words of their own to wait for."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
PROGRAM = """
import ctypes as C
import raccoongpurender_gb300 as rg
from raccoongpurender_gb300 import scenes

lib = rg.load_library()
rt = None
for name in ("libcudart.so.13", "/usr/local/cuda/lib64/libcudart.so.13", "/usr/local/cuda/lib64/libcudart.so"):
    try:
        rt = C.CDLL(name)
        break
    except OSError:
        pass
assert rt is not None
camd = scenes.cornell_camera()
cam = rg.camera_look_at(camd["eye"], camd["target"], camd["up"], camd["vfov"], 24, 20)


def render():
    sm = rg.SceneManager()
    sm.addMesh(scenes.cornell_box())
    sm.buildBVH()
    lane = rg.WavefrontLane(0, 1024)
    lane.setup(sm)
    lane.initialize(cam, rg.render_config(spp=3, max_depth=5))
    steps = lane.render_until_done()
    return steps, lane.accumulation()[..., 3].sum()


first = render()
rg.Guide(0)
assert rt.cudaDeviceReset() == 0
assert render() == first
assert rt.cudaDeviceReset() == 0
keep = [rg.WavefrontLane(0, 1024) for _ in range(70)]
assert render() == first
print("reset ok")
"""


def test_reset(rg):
    root = Path(__file__).resolve().parents[1]
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "reset ok" in r.stdout, r.stdout + r.stderr
