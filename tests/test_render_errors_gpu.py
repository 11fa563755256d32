"""A render whose error word is set (here by a checkpoint that holds it, as one taken after a full
traversal stack would) runs to its end like any other and then reports it; its state is one
that whole bounces leave."""
import struct

import numpy as np
import pytest

from raccoongpurender_gb300 import scenes
from tests.helpers import build, camera

pytestmark = pytest.mark.gpu
HEADER, TILE = 56, 4096


def _parts(pool):
    """(name, bytes) of a checkpoint's state after its header, in order, up to the error word."""
    tiles = -(-pool // TILE)
    n = tiles * TILE
    return [("slots", 128 * n), ("qid", n), ("req", 2 * n), ("counts", 32), ("tile_new", 4 * tiles), ("scalars", 64),
            ("err", 16)]


def _split(state, pool):
    out, at = {}, HEADER
    for name, size in _parts(pool):
        out[name] = bytes(state[at:at + size])
        at += size
    out["scalars"] = out["scalars"][:24]  # next pixel, step base, rays; then the cast's counter
    return out


@pytest.mark.parametrize("persistent", [True, False])
@pytest.mark.parametrize("max_steps", [1000, 11, 5])
def test_flagged_render_ends_whole(rg, po, persistent, max_steps):
    mesh, env, camd = scenes.mixed_scene(level=3, seed=3)
    sm, _ = build(mesh, env=env)
    cam, config, pool = camera(camd, 40, 36), rg.render_config(spp=40, max_depth=6), 5000
    at = HEADER + sum(size for name, size in _parts(pool) if name != "err")

    def lane_of():
        lane = rg.WavefrontLane(0, pool)
        lane.set_render_trace(persistent, 12)
        lane.setup(sm)
        lane.initialize(cam, config)
        return lane

    a = lane_of()
    a.step(2)
    clean = a.checkpoint()
    assert struct.unpack_from("<I", clean, at)[0] == 0
    flagged = clean.copy()
    flagged[at:at + 4] = np.frombuffer(struct.pack("<I", 1), np.uint8)
    a = lane_of()
    a.restore(flagged)
    with pytest.raises(rg.RgrError) as e:
        a.render_until_done(max_steps)
    assert e.value.status == -5  # RGR_E_OVERFLOW
    b = lane_of()
    b.restore(clean)
    steps = b.render_until_done(max_steps)
    assert steps > 16 or steps == max_steps
    assert a.stats().steps == b.stats().steps == 2 + steps
    assert a.stats().error_flags == 1 and b.stats().error_flags == 0
    for more in (0, 3):
        a.step(more)
        b.step(more)
        x, y = _split(a.checkpoint(), pool), _split(b.checkpoint(), pool)
        x.pop("err"), y.pop("err")
        assert x == y
