"""bench.py names the neighbour mode that the engine runs, from the particle
count and the dense window's size."""
import os
import sys

import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), ".."))
import bench  # noqa: E402
import pbf_b200 as P  # noqa: E402
from pbf_b200 import scenes  # noqa: E402


def derived(side, **kw):
    """side^3 cells of h = 0.1 between the walls, (side + 13)^3 in the window."""
    cfg = scenes.base_config(0.1, 0.05, (0.1 * side + 0.05,) * 3, 1, 1, 1.0 / 60.0, 1000)
    for k, v in kw.items():
        setattr(cfg, k, v)
    return P.derive_params(cfg)


@pytest.mark.parametrize("asked,n,side,mode", [
    (-1, (3 << 16) - 1, 20, 4), (-1, 3 << 16, 20, 8), (-1, 3 << 16, 130, 8), (-1, 3 << 16, 140, 4),
    (-1, 3 << 16, 150, 4), (-1, 1 << 18, 145, 8), (-1, 1 << 18, 150, 4), (-1, (1 << 18) + 1, 230, 8), (-1, (1 << 18) + 1, 250, 4), (-1, 1 << 19, 250, 8),
    (-1, 1 << 22, 390, 8), (-1, 1 << 22, 400, 4), (8, 100, 20, 8), (8, 100, 400, 4), (4, 1 << 22, 20, 4),
    (8, 1 << 27, 20, 4)])
def test_mode(asked, n, side, mode):
    assert bench.neighbour_mode(asked, n, derived(side)) == mode


def test_apbf_runs_the_buckets():
    assert bench.neighbour_mode(8, 1 << 20, derived(20, enable_apbf=1)) == 4
