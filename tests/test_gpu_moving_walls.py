"""Walls that cross cells: below 2^19 particles the automatic neighbour mode
does not make a dense window's tables anew step after step, follows a window
that has settled, and gives the bits of either mode throughout."""
import numpy as np
import pytest

import pbf_b200 as P
from test_gpu_coop import moving_block

pytestmark = pytest.mark.gpu

N = 200000
CELL = 0.04


@pytest.mark.parametrize("graph", [False, True])
def test_windows_that_change(have_gpu, graph):
    cfg, pos, vel = moving_block(N, 0.02, CELL, 1)
    cfg.solver_iterations = 2
    box = np.array(cfg.bounds_max[:])
    # cells the far walls stand out by: still, moving every step, still, moving every 6th step
    out = [0] * 3 + [1, 2, 3, 4, 3, 2] + [2] * 6 + [3] * 6 + [4] * 2
    dense = []
    got = []
    for mode in (-1, 4, 8):
        fl = P.PBFluids(cfg)
        fl.set_option(1, mode)
        fl.set_use_graph(graph)
        fl.setParticles(P.make_particles(pos, vel))
        for k in out:
            fl.setBounds((0, 0, 0), tuple(box + k * CELL), cfg.bound_damping)
            fl.step()
            if mode < 0:
                dense.append(any(fl.list_stats()))
        got.append(fl.readbackParticles())
    # the first change is followed, those right after it are not, nor the still window before its fourth step
    want = [True] * 3 + [True] + [False] * 5 + [False] * 3 + [True] * 3 + [True] * 6 + [True] * 2
    assert dense == want
    for g in got[1:]:
        assert np.array_equal(g["pos"], got[0]["pos"]) and np.array_equal(g["vel"], got[0]["vel"])
