"""Stages run out of their order: a delta-p stage replays a lambda stage's
hits only when that lambda ran in the same iteration on the same positions,
table and radius; otherwise it walks the cells, whatever number the iteration
has (0 is pbf_run_stage's own default)."""
import numpy as np
import pytest

import pbf_b200 as P
from test_gpu_coop import moving_block

pytestmark = pytest.mark.gpu

SORTED = (P.STAGE_PREDICT, P.STAGE_SORT, P.STAGE_TABLE, P.STAGE_REORDER)
NEVER = 77  # no lambda stage ran in this iteration


def prepared(n, mode, h=0.04):
    """A scene after two steps, whose second left other positions and hits."""
    cfg, pos, vel = moving_block(n, 0.02, h, 3)
    fl = P.PBFluids(cfg)
    fl.set_option(1, mode)
    fl.setParticles(P.make_particles(pos, vel))
    fl.step()
    fl.step()
    fl.uploadParticles(P.make_particles(pos[::-1].copy(), vel))
    return fl, cfg


def after(n, mode, stages):
    fl, _ = prepared(n, mode)
    for s in stages:
        fl.run_stage(*s)
    return fl.read_buffer(P.BUF_XSTAR, np.float32, (n, 4))


@pytest.mark.parametrize("mode", [4, 8])
@pytest.mark.parametrize("n", [600, 6000, 20000])
def test_deltap_without_lambda_walks(have_gpu, n, mode):
    head = [(s,) for s in SORTED]
    walked = after(n, mode, head + [(P.STAGE_DELTAP, NEVER)])
    assert np.isfinite(walked).all()
    for it in (0, 1, 0xFFFFFFFF):
        assert np.array_equal(after(n, mode, head + [(P.STAGE_DELTAP, it)]), walked)


@pytest.mark.parametrize("mode", [4, 8])
@pytest.mark.parametrize("n", [600, 6000, 20000])
def test_replayed_and_walked_hits_are_the_same(have_gpu, n, mode):
    for it in (0, 1, 0xFFFFFFFF):
        head = [(s,) for s in SORTED] + [(P.STAGE_LAMBDA, it)]
        assert np.array_equal(after(n, mode, head + [(P.STAGE_DELTAP, it)]), after(n, mode, head + [(P.STAGE_DELTAP, NEVER)]))


@pytest.mark.parametrize("n", [600, 20000])
def test_hits_do_not_outlive_the_radius(have_gpu, n):
    got = []
    for it in (1, NEVER):
        fl, cfg = prepared(n, 4)
        for s in SORTED:
            fl.run_stage(s)
        fl.run_stage(P.STAGE_LAMBDA, 1)
        cfg.h = 0.05
        cfg.hash_size = fl.params().hash_size
        fl.setParams(cfg)
        fl.run_stage(P.STAGE_DELTAP, it)
        got.append(fl.read_buffer(P.BUF_XSTAR, np.float32, (n, 4)))
    assert np.array_equal(*got)
