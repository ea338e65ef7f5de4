"""Stages before those whose results they read: a permutation or a table that
is not there, or no longer fits the particles, is an error or empty, never
what the memory happened to hold."""
import numpy as np
import pytest

import pbf_b200 as P
from test_gpu_coop import moving_block

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [4, 8])
def test_growing_drops_the_permutation(have_gpu, mode):
    cfg, pos, vel = moving_block(4000, 0.02, 0.04, 1)
    fl = P.PBFluids(cfg)
    fl.set_option(1, mode)
    fl.setParticles(P.make_particles(pos[:500], vel[:500]))
    fl.step()
    fl.setParticles(P.make_particles(pos, vel))
    for st in (P.STAGE_TABLE, P.STAGE_REORDER, P.STAGE_LAMBDA, P.STAGE_DELTAP):
        with pytest.raises(P.PBFError):
            fl.run_stage(st, 1)
    for which in (P.BUF_SORTED_IDS, P.BUF_SORTED_KEYS):
        with pytest.raises(P.PBFError):
            fl.read_buffer(which, np.uint32, 4000)


def test_passes_without_a_table_meet_nobody(have_gpu):
    n = 3000
    cfg, pos, vel = moving_block(n, 0.02, 0.04, 1)
    cfg.substep_iterations = 1
    fl = P.PBFluids(cfg)
    fl.set_option(1, 4)
    fl.setParticles(P.make_particles(pos, vel))
    for st in (P.STAGE_PREDICT, P.STAGE_SORT, P.STAGE_REORDER):
        fl.run_stage(st)
    x = fl.read_buffer(P.BUF_XSTAR, np.float32, (n, 4))
    fl.run_stage(P.STAGE_LAMBDA, 1)
    fl.run_stage(P.STAGE_DELTAP, 1)
    assert np.array_equal(fl.read_buffer(P.BUF_XSTAR, np.float32, (n, 4))[:, :3], x[:, :3])
    assert (fl.read_buffer(P.BUF_TABLE, np.int32, (cfg.hash_size, 2)) == -1).all()
