"""The byte count behind bench.py's render roofline: what the kernels of a bounce inside a run
use, no logic pass."""
import pytest

import bench


def test_state_bytes():
    # a path that goes on, in a volume: shading 238, cast 101, classification 5
    assert bench.render_state_bytes(0.0, 1.0, 0.0) == 238 + 101 + 5
    assert bench.render_state_bytes(0.0, 0.0, 0.0) == 206 + 101 + 5
    # one that ends: its new path takes its place
    assert bench.render_state_bytes(1.0, 0.0, 0.0) == 202 + 101 + 3
    assert bench.render_state_bytes(0.25, 0.5, 0.25) == pytest.approx(
        101 + 1 + 0.5 + 3.0 + 0.25 * 202 + 0.75 * (206 + 16 + 8))
