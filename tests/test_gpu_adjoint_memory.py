"""The adjoint with less and less free device memory: a record of every
substep, one record that the backward fills again, and one without hits, whose
passes walk the buckets.  The gradients are the same up to the order of the
atomic sums, and the last takes what the checkpoints, the iterations' (x*,
lambda), denominators and raw dp and the adjoints take."""
import numpy as np
import pytest
import torch

from adjoint_cases import setup
from test_gpu_adjoint import gpu_grads, make_batch, rel

pytestmark = pytest.mark.gpu

MB = 1 << 20


def run(b, pos, vel, target, offs):
    free0 = torch.cuda.mem_get_info()[0]
    out = gpu_grads(b, pos, vel, target, offs)
    torch.cuda.synchronize()
    return out, free0 - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("nside,copies", [(26, 4), (26, 16)])
def test_gradients_at_every_size_of_record(have_gpu, nside, copies):
    subs, iters = 3, 2
    cfg, _, pos, vel, grid, target = setup(nside=nside, subs=subs, iters=iters, scorr=False)
    cfg.bounds_max[:] = [1.5, 1.5, 1.5]
    n = len(pos) * copies
    offs = np.zeros((copies, 3))
    hits = n * 4 * 65 * (iters + 1)             # bytes of one record's hits
    rest = n * (52 * iters + 52)                # and of its other arrays
    lean = n * (32 * subs + 160 + 52 * iters)   # what the smallest kind takes
    torch.cuda.empty_cache()
    first, held = run(make_batch(cfg, pos, vel, grid, copies), pos, vel, target, offs)
    assert held >= subs * (hits + rest)
    # less than four times all records, then less than twice one
    for limit, most in ((3 * subs * (hits + rest), lean + 2 * (hits + rest)), ((hits + rest) // 2, lean)):
        b = make_batch(cfg, pos, vel, grid, copies)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        # (room for the checkpoints and adjoints beside the limit, and for what a graph takes)
        keep = limit + lean + 48 * MB
        hog = torch.empty(torch.cuda.mem_get_info()[0] - keep, dtype=torch.uint8, device="cuda")
        try:
            got, held = run(b, pos, vel, target, offs)
        finally:
            del hog
            torch.cuda.empty_cache()
        assert held <= most + 96 * MB
        assert rel(got[0], first[0]) <= 1e-5 and rel(got[1], first[1]) <= 1e-5 and rel(got[2], first[2]) <= 1e-4
        assert np.array_equal(got[3], first[3])
        del b
