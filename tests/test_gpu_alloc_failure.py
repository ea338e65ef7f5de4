"""A scene that does not fit: the call says so, the handle holds no particles,
and takes the next scene as a fresh one does."""
import numpy as np
import pytest
import torch

import pbf_b200 as P
from pbf_b200._capi import lib
from test_gpu_coop import moving_block, stepped

pytestmark = pytest.mark.gpu

TOO_MANY = 2_000_000_000  # some 800 GB of arrays


@pytest.mark.parametrize("mode", [4, 8])
@pytest.mark.parametrize("graph", [False, True])
def test_scene_too_large(have_gpu, mode, graph):
    cfg, pos, vel = moving_block(900, 0.02, 0.04, 1)
    want = stepped(cfg, pos, vel, mode)
    fl = P.PBFluids(cfg)
    fl.set_option(1, mode)
    fl.set_use_graph(graph)
    fl.setParticles(P.make_particles(pos, vel))
    fl.step()
    some = torch.zeros(16, device="cuda")
    rc = lib().pbf_set_particles_device(fl.handle, some.data_ptr(), some.data_ptr(), TOO_MANY)
    assert rc == -4  # PBF_ERR_ALLOC
    fl.step()  # nothing to do
    with pytest.raises(P.PBFError):
        fl.run_stage(P.STAGE_PREDICT)
    fl.setParticles(P.make_particles(pos, vel))
    fl.step()
    fl.step()
    got = fl.readbackParticles()
    assert np.array_equal(got["pos"], want["pos"]) and np.array_equal(got["vel"], want["vel"])
