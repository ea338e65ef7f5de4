"""An SDF grid that does not fit: the call says so and the scene goes on
without an obstacle, as after its removal."""
import ctypes as C

import numpy as np
import pytest
import torch

import pbf_b200 as P
from pbf_b200._capi import lib
from test_gpu_coop import moving_block

pytestmark = pytest.mark.gpu

DIMS = (1024, 1024, 512)  # 2 GB


def small_grid():
    x = np.stack(np.meshgrid(*[np.arange(12) * 0.05] * 3, indexing="ij"), -1)
    return (np.linalg.norm(x - 0.2, axis=-1) - 0.1).astype(np.float32)


def refused(call, handle, *head):
    """The call with a grid larger than what is free (which nobody reads)."""
    grid = np.empty(DIMS, np.float32)
    torch.cuda.synchronize()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (512 << 20), dtype=torch.uint8, device="cuda")
    try:
        return call(handle, *head, grid.ctypes.data_as(C.c_void_p), (C.c_int32 * 3)(*DIMS), (C.c_float * 3)(0, 0, 0),
                    C.c_float(0.1))
    finally:
        del hog
        torch.cuda.empty_cache()


@pytest.mark.parametrize("graph", [False, True])
def test_scene(have_gpu, graph):
    cfg, pos, vel = moving_block(900, 0.02, 0.04, 1)
    out = []
    for fail in (False, True):
        sdf = P.GridSDF(small_grid(), (0, 0, 0), 0.05)
        fl = P.PBFluids(cfg)
        fl.set_use_graph(graph)
        fl.setParticles(P.make_particles(pos, vel))
        fl.setSDFBoundary(sdf)
        fl.step()
        if fail:
            assert refused(lib().pbf_set_sdf_grid, sdf._h) == -4
        else:
            fl.setSDFBoundary(None)
        fl.step()
        out.append(fl.readbackParticles())
    assert np.array_equal(out[0]["pos"], out[1]["pos"]) and np.array_equal(out[0]["vel"], out[1]["vel"])


@pytest.mark.parametrize("graph", [0, 1])
def test_batch(have_gpu, graph):
    cfg, pos, vel = moving_block(900, 0.02, 0.04, 1)
    out = []
    for fail in (False, True):
        b = P.Batch(cfg, [dict(n=len(pos), bounds_min=tuple(cfg.bounds_min), bounds_max=tuple(cfg.bounds_max),
                               hash_size=cfg.hash_size)] * 2)
        b.set_option(P.BOPT_USE_GRAPH, graph)
        for k in range(2):
            b.set_particles(k, P.make_particles(pos, vel))
            b.set_sdf_grid(k, small_grid(), (0, 0, 0), 0.05)
        b.step()
        if fail:
            assert refused(lib().pbf_batch_set_sdf_grid, b.handle, 1) == -4
        else:
            b.clear_sdf(1)
        b.step()
        out.append(b.read_particles())
    assert np.array_equal(out[0]["pos"], out[1]["pos"]) and np.array_equal(out[0]["vel"], out[1]["vel"])
