"""Neighbour passes with a group of lanes per particle (k_coop.cu) against the
dense-window passes (k_dense.cu), which walk the same pairs in another way:
bit-identical.  Sizes at the edges of the group widths (32, 16 and 8 lanes,
then one thread), buckets of more candidates than a group lists at a time and
more hits than it keeps, and every s_corr branch."""
import numpy as np
import pytest

import pbf_b200 as P
from pbf_b200 import scenes

pytestmark = pytest.mark.gpu


def moving_block(n, d, h, seed, hash_size=None):
    side = int(np.ceil(n ** (1.0 / 3.0)))
    rng = np.random.default_rng(seed)
    pos = scenes.lattice(side, side, side, d, (0.0, 0.0, 0.0), 0.0, 0)[:n]
    pos = np.clip(pos + rng.uniform(-0.2 * d, 0.2 * d, pos.shape), 1e-4, None).astype(np.float32)
    vel = (rng.normal(size=pos.shape) * 0.1 * d * 120.0).astype(np.float32)
    box = 1.5 * side * d
    cfg = scenes.base_config(h, d, (box, box, box), 2, 3, 1.0 / 60.0, n, hash_size)
    return cfg, pos, vel


def stepped(cfg, pos, vel, mode, steps=2):
    fl = P.PBFluids(cfg)
    fl.set_option(1, mode)
    fl.setParticles(P.make_particles(pos, vel))
    for _ in range(steps):
        fl.step()
    return fl.readbackParticles()


def same(a, b):
    return np.array_equal(a["pos"], b["pos"]) and np.array_equal(a["vel"], b["vel"])


@pytest.mark.parametrize("n", [1, 2, 33, 1000, 4096, 4097, 8192, 8193, 1 << 18, (1 << 18) + 1])
def test_group_widths_are_bit_identical_to_dense_windows(have_gpu, n):
    cfg, pos, vel = moving_block(n, 0.02, 0.04, n)
    assert same(stepped(cfg, pos, vel, 4), stepped(cfg, pos, vel, 8))


@pytest.mark.parametrize("n", [3000, 6000, 9000])
@pytest.mark.parametrize("d,hash_size", [(0.02, 64), (0.011, 1 << 15), (0.011, 16)])
def test_long_buckets_and_many_hits(have_gpu, n, d, hash_size):
    """64 buckets of a hundred particles and more, 200 hits a particle."""
    cfg, pos, vel = moving_block(n, d, 0.04, 7, hash_size)
    assert same(stepped(cfg, pos, vel, 4, 1), stepped(cfg, pos, vel, 8, 1))


@pytest.mark.parametrize("n", [2000, 6000, 12000])
@pytest.mark.parametrize("change", [dict(enable_scorr=0), dict(n_corr=3.0), dict(enable_viscosity=0),
                                    dict(enable_vorticity=0), dict(enable_viscosity=0, enable_vorticity=0)])
def test_options(have_gpu, n, change):
    cfg, pos, vel = moving_block(n, 0.02, 0.04, 11)
    for k, v in change.items():
        setattr(cfg, k, v)
    assert same(stepped(cfg, pos, vel, 4), stepped(cfg, pos, vel, 8))


@pytest.mark.parametrize("sizes", [[1], [700, 1, 1500], [3000, 5200, 4100], [70000, 1, 131000]])
def test_batches(have_gpu, sizes):
    from pbf_b200 import batch as PB
    cfg, sc = scenes.c3(5, len(sizes), sizes)
    out = []
    for mode in (4, 8):
        b = PB.make_batch(cfg, sc)
        b.set_option(P.BOPT_NEIGHBOUR_MODE, mode)
        for _ in range(2):
            b.step()
        out.append(b.read_particles())
    assert same(*out)


def test_coincident_particles(have_gpu):
    """r = 0 pairs: density without a gradient."""
    cfg, pos, vel = moving_block(3000, 0.02, 0.04, 13)
    pos[1::2] = pos[::2]
    vel[1::2] = vel[::2]
    assert same(stepped(cfg, pos, vel, 4), stepped(cfg, pos, vel, 8))


@pytest.mark.parametrize("n,hash_size", [(1, 1), (3, 2), (300, 1), (300, 4), (5000, 4096), (5000, 8192), (5000, 1 << 21),
                                         (5000, 1 << 22), (70000, 1 << 17)])
def test_sort_of_a_step_equals_the_stages(have_gpu, n, hash_size):
    """A step's own sort (k_bucket.cu) leaves the keys, permutation and table
    that the stages one by one leave, for tables of one bucket to more than it
    takes, and the same state."""
    cfg, pos, vel = moving_block(n, 0.02, 0.04, n, hash_size)
    cfg.substep_iterations = 1
    got = []
    for stages in (False, True):
        fl = P.PBFluids(cfg)
        fl.set_option(1, 4)
        fl.setParticles(P.make_particles(pos, vel))
        for _ in range(2):
            if stages:
                for st in (P.STAGE_PREDICT, P.STAGE_SORT, P.STAGE_TABLE, P.STAGE_REORDER):
                    fl.run_stage(st)
                for it in range(1, cfg.solver_iterations + 1):
                    fl.run_stage(P.STAGE_LAMBDA, it)
                    fl.run_stage(P.STAGE_DELTAP, it)
                fl.run_stage(P.STAGE_INTEGRATE)
                fl.run_stage(P.STAGE_VORTICITY)
            else:
                fl.step()
        fl.sync()
        got.append([fl.read_buffer(P.BUF_KEYS, np.uint32, n), fl.read_buffer(P.BUF_SORTED_KEYS, np.uint32, n),
                    fl.read_buffer(P.BUF_SORTED_IDS, np.uint32, n), fl.read_buffer(P.BUF_TABLE, np.int32, (hash_size, 2)),
                    fl.read_buffer(P.BUF_XSTAR, np.float32, (n, 4)), fl.readbackParticles()])
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [1, 15, 17, 600, 25000])
@pytest.mark.parametrize("fast", [False, True])
def test_bucket_walkers_of_a_dense_window(have_gpu, n, fast):
    """Particles along the box's near-zero edges, whose cells meet exact hash
    collisions: all of them walk buckets, in a large window of clean cells (one
    group of lanes each), up to more than the list of a launch holds; `fast`
    ones leave the window in between."""
    rng = np.random.default_rng(n)
    h, box = 0.04, 3.0
    pos = rng.uniform(0.0, 1.0, (n, 3)) * [2 * h, 2 * h, box]
    turn = rng.integers(0, 3, n)
    pos = np.stack([np.take_along_axis(pos, ((k + turn) % 3)[:, None], 1)[:, 0] for k in range(3)], 1).astype(np.float32)
    vel = rng.normal(size=(n, 3)).astype(np.float32)
    if fast:
        vel[::3] *= 200.0
    cfg = scenes.base_config(h, h / 2, (box, box, box), 2, 3, 1.0 / 60.0, n, 1 << 16)
    assert same(stepped(cfg, pos, vel, 4), stepped(cfg, pos, vel, 8))


@pytest.mark.parametrize("n,hash_size", [(1, 1), (3, 2), (200, 4), (255, 8), (5000, 128), (5000, 1 << 14), (70001, 1 << 17),
                                         (1 << 20, 1 << 18), ((1 << 20) + 1, 1 << 18)])
def test_sort_of_a_dense_step_equals_the_stages(have_gpu, n, hash_size):
    """The same for dense windows (k_d_sort_*), up to one particle more than it
    takes, with cells outside the window."""
    cfg, pos, vel = moving_block(n, 0.02, 0.04, n, hash_size)
    vel[::7] *= 100.0
    cfg.substep_iterations = 1
    got = []
    for stages in (False, True):
        fl = P.PBFluids(cfg)
        fl.set_option(1, 8)
        fl.setParticles(P.make_particles(pos, vel))
        for _ in range(2):
            if stages:
                for st in (P.STAGE_PREDICT, P.STAGE_SORT, P.STAGE_TABLE, P.STAGE_REORDER):
                    fl.run_stage(st)
                for it in range(1, cfg.solver_iterations + 1):
                    fl.run_stage(P.STAGE_LAMBDA, it)
                    fl.run_stage(P.STAGE_DELTAP, it)
                fl.run_stage(P.STAGE_INTEGRATE)
                fl.run_stage(P.STAGE_VORTICITY)
            else:
                fl.step()
        fl.sync()
        got.append([fl.read_buffer(P.BUF_KEYS, np.uint32, n), fl.read_buffer(P.BUF_SORTED_KEYS, np.uint32, n),
                    fl.read_buffer(P.BUF_SORTED_IDS, np.uint32, n), fl.read_buffer(P.BUF_TABLE, np.int32, (hash_size, 2)),
                    fl.read_buffer(P.BUF_XSTAR, np.float32, (n, 4)), fl.readbackParticles()])
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("hash_size", [16, 128, 1 << 14])
def test_sort_of_a_dense_batch(have_gpu, hash_size):
    """A batch's sort by counting, and by radix where a scene's buckets are too
    long for it, with particles that leave their scene's window."""
    from pbf_b200 import batch as PB
    cfg, sc = scenes.c3(5, 4, [5000, 1, 300, 8000])
    for k, s in enumerate(sc):
        s["hash_size"] = hash_size
        s["vel"] = np.array(s["vel"], np.float32)
        s["vel"][k::5] += np.float32(60.0)
    out = []
    for mode in (4, 8):
        b = PB.make_batch(cfg, sc)
        b.set_option(P.BOPT_NEIGHBOUR_MODE, mode)
        for _ in range(2):
            b.step()
        out.append(b.read_particles())
    assert same(*out)
