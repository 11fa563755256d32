"""Closest hits of host arrays into every kind of memory that the call takes: ordinary pages,
which the host brings in beside the kernel, and page-locked, managed and device memory, which
are left alone."""
import ctypes as C

import numpy as np
import pytest

from raccoongpurender_gb300 import scenes
from tests.conftest import bits
from tests.helpers import build

pytestmark = pytest.mark.gpu
N = 300_000


def _runtime():
    for name in ("libcudart.so.13", "/usr/local/cuda/lib64/libcudart.so.13", "/usr/local/cuda/lib64/libcudart.so"):
        try:
            return C.CDLL(name)
        except OSError:
            continue
    pytest.skip("no CUDA runtime library to allocate from")


@pytest.mark.parametrize("kind", ["ordinary", "pinned", "managed", "device"])
def test_results_in_any_memory(rg, po, kind):
    import torch
    torch.zeros(1, device="cuda")
    rt = _runtime()
    sm, osc = build(scenes.displaced_icosphere(4, seed=7))
    lane = rg.WavefrontLane(0, 1024)
    lane.setup(sm)
    rays = scenes.random_rays(N, (-1.3, -1.3, -1.3), (1.3, 1.3, 1.3), seed=2)
    oprim, ot, _ = osc.trace(rays.packed8(), threads=16)
    keep, out = [], []
    for _ in range(2):
        p = C.c_void_p()
        if kind == "ordinary":
            keep.append(np.zeros(4 * N, np.uint8))
            p.value = keep[-1].ctypes.data
        elif kind == "pinned":
            assert rt.cudaHostAlloc(C.byref(p), C.c_size_t(4 * N), C.c_uint(0)) == 0
        elif kind == "managed":
            assert rt.cudaMallocManaged(C.byref(p), C.c_size_t(4 * N), C.c_uint(1)) == 0
        else:
            assert rt.cudaMalloc(C.byref(p), C.c_size_t(4 * N)) == 0
        out.append(p)
    soa = [np.ascontiguousarray(a, np.float32) for a in rays.soa()]
    r = rg.rgr_ray_soa(*[rg._ptr(a) for a in soa])
    for _ in range(2):
        assert lane._lib.rgr_trace_closest(lane._h, C.byref(r), N, out[0], out[1]) == 0
        prim, t = np.empty(N, np.int32), np.empty(N, np.float32)
        for dst, src in ((prim, out[0]), (t, out[1])):
            assert rt.cudaMemcpy(dst.ctypes.data_as(C.c_void_p), src, C.c_size_t(4 * N), C.c_int(4)) == 0
        assert (prim == oprim).all() and (bits(t) == bits(ot)).all()
    if kind == "pinned":
        [rt.cudaFreeHost(p) for p in out]
    elif kind in ("managed", "device"):
        [rt.cudaFree(p) for p in out]
