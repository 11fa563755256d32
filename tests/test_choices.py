"""The rules by which calls choose their kernels (csrc/host/choices.h, plain C++),
compiled and called on the host."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "raccoongpurender_gb300" / "csrc"
WRAP = """
#include "host/choices.h"
extern "C" int persistent(int mode, uint64_t pool, uint64_t samples) {
    return rgr::persistent_cast(mode, pool, samples);
}
extern "C" uint32_t half_end(uint64_t pool, uint64_t samples, uint32_t resident, uint32_t tile) {
    return rgr::cast_half_end(pool, samples, resident, tile);
}
extern "C" int per_slot(uint32_t prims) { return rgr::per_slot_cast(prims); }
extern "C" void tuning(int refill, int search, int* out) {  // 0: not set
    rgr::CastTuning t;
    if (refill) rgr::set_refill(t, 31), rgr::set_refill(t, refill);
    if (search) rgr::set_search(t, 31), rgr::set_search(t, search);
    out[0] = t.refill, out[1] = t.search, out[2] = t.mixed_refill, out[3] = t.mixed_search;
}
extern "C" int shade_blocks() { return rgr::kShadeBlocksPerSm; }
extern "C" void grids(int sms, int blocks, int staged, int plain, int* out) {
    const rgr::TraceGrids g = rgr::trace_grids(sms, blocks, staged, plain);
    out[0] = g.staged, out[1] = g.plain;
}
extern "C" uint32_t blocks(uint64_t pool, uint32_t half_end) { return rgr::cast_blocks(pool, half_end); }
"""


@pytest.fixture(scope="module")
def choices(tmp_path_factory):
    d = tmp_path_factory.mktemp("choices")
    (d / "wrap.cpp").write_text(WRAP)
    r = subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-shared", "-fPIC", f"-I{CSRC}", str(d / "wrap.cpp"),
                        "-o", str(d / "choices.so")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(str(d / "choices.so"))


@pytest.mark.parametrize("pool,samples,persistent", [
    (3 << 17, 0, 1), ((3 << 17) - 1, 0, 0), (1 << 24, 0, 1),  # no budget: the pool counts
    (649316, 20440, 0),                                       # a small image in a large pool
    (1 << 24, (3 << 17) - 1, 0), (1 << 24, 3 << 17, 1),
    (1 << 18, 1 << 30, 0), (1 << 20, 1 << 40, 1),
])
def test_cast_by_paths_in_flight(choices, pool, samples, persistent):
    f = choices.persistent
    assert f(-1, C.c_uint64(pool), C.c_uint64(samples)) == persistent
    assert f(1, C.c_uint64(pool), C.c_uint64(samples)) == 1
    assert f(0, C.c_uint64(pool), C.c_uint64(samples)) == 0


@pytest.mark.parametrize("pool", [1, 255, 256, 257, 4096, 4097, 20000, 155648, 155649, 160000, 649316])
@pytest.mark.parametrize("samples", [0, 1, 2880, 4096, 4097, 20440, 155648, 155649, 1 << 40])
def test_fused_blocks_cover_the_pool(choices, pool, samples):
    """Every slot in one block, each block's slots in one tile; halves only while the paths in
    flight fill no more than a wave of 608 blocks."""
    span, tile = 512, 4096
    half_end = choices.half_end(C.c_uint64(pool), C.c_uint64(samples), 608, tile)
    inflight = min(pool, samples) if samples else pool
    assert half_end == (-(-inflight // tile) * tile if inflight <= 256 * 608 else 0)
    at = 0
    for b in range(choices.blocks(C.c_uint64(pool), half_end)):  # as k_cast_logic finds its slots
        half_blocks = half_end // (span // 2)
        n = span // 2 if b < half_blocks else span
        first = b * (span // 2) if b < half_blocks else half_end + (b - half_blocks) * span
        assert first == at and first // tile == (first + n - 1) // tile
        at += n
    assert pool <= at < pool + span


def test_small_scenes_cast_per_slot(choices):
    assert [choices.per_slot(n) for n in (0, 36, 1024, 1025, 1 << 27)] == [1, 1, 1, 0, 0]


def test_tuned_thresholds(choices):
    """A caller who sets the defaults has the library's own thresholds, for warps of one octant and
    of several; so has the autotuner's first trial."""
    from raccoongpurender_gb300 import autotune

    def tuning(refill, search):
        out = (C.c_int * 4)()
        choices.tuning(refill, search, out)
        return tuple(out)

    untouched = tuning(0, 0)
    assert untouched == (24, 8, 12, 12)
    d = autotune.TRACE_DEFAULTS
    assert tuning(d["trace_refill"], d["trace_search"]) == untouched
    assert tuning(16, 0) == (16, 8, 16, 12) and tuning(0, 4) == (24, 4, 12, 4)
    assert tuning(12, 12) == (12, 12, 12, 12) and tuning(32, 1) == (32, 1, 32, 1)


def test_defaults_agree(choices):
    """The Python setters called without arguments, and the autotuner's starting points, are what
    the library does untouched."""
    import inspect

    import raccoongpurender_gb300 as rg
    from raccoongpurender_gb300 import autotune

    def default(f, name):
        return inspect.signature(f).parameters[name].default

    out = (C.c_int * 4)()
    choices.tuning(0, 0, out)
    refill, search = out[0], out[1]
    blocks = choices.shade_blocks()
    for cls in (rg.WavefrontLane, rg.Batch):
        assert default(cls.set_render_tuning, "shade_blocks_per_sm") == blocks
        assert default(cls.set_render_tuning, "graph_steps") == 1  # rgr_context's graph_steps_default
        assert default(cls.set_render_trace, "refill") == autotune.DEFAULTS["render_refill"] == 12
        assert default(cls.set_render_trace, "persistent") == -1
        assert default(cls.set_trace_search, "render") == autotune.DEFAULTS["render_search"] == 8
    assert autotune.DEFAULTS["shade_blocks"] == blocks
    assert default(rg.WavefrontLane.set_trace_tuning, "refill") == refill
    assert default(rg.WavefrontLane.set_trace_search, "closest") == search


@pytest.mark.parametrize("blocks,staged,plain,want", [
    (0, 5, 5, (760, 760)),
    (0, 2, 5, (304, 760)),  # staged nodes leave room for fewer blocks; calls that stage none keep theirs
    (3, 2, 5, (304, 456)), (2, 3, 5, (304, 304)),
])
def test_grids(choices, blocks, staged, plain, want):
    out = (C.c_int * 2)()
    choices.grids(152, blocks, staged, plain, out)
    assert tuple(out) == want
