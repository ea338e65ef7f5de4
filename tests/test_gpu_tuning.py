"""The batch autotuner where block, order and persistence shape no pass: a
small batch's neighbour passes take a group of lanes per particle whatever
they are, so mode 4 has one speed and the settings stay as they were."""
import pytest

import pbf_b200 as P
from pbf_b200 import batch as PB
from pbf_b200 import scenes

pytestmark = pytest.mark.gpu


def test_shapes_that_do_not_matter_are_timed_once(have_gpu):
    cfg, sc = scenes.c3(5, 3, [900, 400, 1300])
    b = PB.make_batch(cfg, sc)
    b.set_option(P.BOPT_NEIGHBOUR_MODE, 4)
    b.set_option(P.BOPT_BLOCK, 256)
    b.set_option(P.BOPT_BLOCKS_PER_SM, 3)
    b.step()
    before = b.kernel_launches()
    b.step()
    step = b.kernel_launches() - before
    best, cands = b.autotune(4)
    assert len(cands) == 12 and len({c["ms_per_step"] for c in cands}) == 1
    assert b.kernel_launches() - before - step <= 5 * step  # one warm-up and four trial steps
    assert (best["block"], best["order"], best["blocks_per_sm"]) == (256, 1, 3)
    assert (b.get_option(P.BOPT_BLOCK), b.get_option(P.BOPT_BLOCKS_PER_SM)) == (256, 3)
