"""Requests that share a pool, with the cast and the bounces that large pools take (and those of
small ones): against the oracle whatever number of bounces lies between two looks at the
outcome, and where the bounces end inside a run."""
import numpy as np
import pytest

import raccoongpurender_gb300 as rg
from tests import test_batch_gpu
from tests.helpers import compare_slots
from tests.test_batch_gpu import _requests

pytestmark = pytest.mark.gpu
FIELDS = ["T", "L", "ro", "rd", "rng", "pixel_index", "queue"]


@pytest.mark.parametrize("persistent", [True, False])
@pytest.mark.parametrize("steps_per_launch,max_steps", [(1, 1000), (4, 1000), (8, 1000), (5, 11), (1, 3), (8, 8)])
@pytest.mark.parametrize("order", [rg.ORDER_FIFO, rg.ORDER_SHORTEST_FIRST])
def test_runs_match_the_oracle(po, persistent, steps_per_launch, max_steps, order):
    reqs = _requests(po)
    npaths = (1 << 12) + 77
    b = rg.Batch(0, npaths)
    b.set_render_trace(12, persistent)
    ids = [b.add(sm, cam, cfg) for sm, _, cam, cfg in reqs]
    if max_steps < 1000:
        with pytest.raises(rg.RgrError) as e:  # not all requests are finished
            b.run(order=order, steps_per_launch=steps_per_launch, max_steps=max_steps)
        assert e.value.status == -4
        steps = -(-max_steps // steps_per_launch) * steps_per_launch  # whole groups
    else:
        steps = b.run(order=order, steps_per_launch=steps_per_launch)
        assert steps > 16 and steps % steps_per_launch == 0
    run_order = sorted(ids, key=lambda i: b.request_stats(i).order)
    oaccs, oslots = po.render_batch([reqs[i][1] for i in run_order],
                                    [po.camera_from_rgr(reqs[i][2]) for i in run_order],
                                    [po.config_from_rgr(reqs[i][3], reqs[i][2].image_w * reqs[i][2].image_h)
                                     for i in run_order], npaths, steps, threads=16)
    assert compare_slots(b.debug_slots(), oslots, fields=FIELDS) == {}
    flight = oslots["queue"] > 0  # in a material queue (0: ended, -1: retired)
    for k, i in enumerate(run_order):
        ga, oa = b.accumulation(i).reshape(-1, 4), oaccs[k]
        assert (ga[:, 3] == oa[:, 3]).all(), f"request {i}"
        np.testing.assert_allclose(ga[:, :3], oa[:, :3], rtol=1e-12, atol=1e-300)
        ms = b.request_stats(i).complete_ms
        if max_steps == 1000:
            assert not flight.any() and 0 < ms < 60e3
        else:
            assert ms == -1.0 or ms > 0
    if max_steps == 1000 and order == rg.ORDER_FIFO:
        # the first request has handed out its samples before the third begins its own
        assert b.request_stats(run_order[0]).complete_ms <= b.request_stats(run_order[2]).complete_ms


def test_unfinished_requests_agree(po):
    """Which requests are finished, and stamped, after a number of bounces does not depend on
    how they are cast."""
    for steps in (6, 12, 20):
        done = []
        for persistent in (True, False):
            b = rg.Batch(0, 1 << 12)
            b.set_render_trace(12, persistent)
            ids = [b.add(sm, cam, cfg) for sm, _, cam, cfg in _requests(po)]
            try:
                b.run(order=rg.ORDER_SHORTEST_FIRST, steps_per_launch=3, max_steps=steps)
            except rg.RgrError as e:
                assert e.status == -4
            done.append([b.request_stats(i).complete_ms > 0 for i in ids])
        assert done[0] == done[1]


def test_eight_requests_persistent(po, monkeypatch):
    """The oracle test of eight requests of 1.5 K to 1.2M triangles, with the cast of large pools."""
    class Persistent(rg.Batch):
        def __init__(self, *args):
            super().__init__(*args)
            self.set_render_trace(12, True)

    monkeypatch.setattr(rg, "Batch", Persistent)
    test_batch_gpu.test_eight_uneven_requests_with_a_million_triangle_scene(po)
