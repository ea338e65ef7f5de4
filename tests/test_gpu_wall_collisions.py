"""Particles predicted cells beyond a wall and clamped back next to resting
ones, where the cell they were predicted in shares its hash bucket with a
neighbour cell of those at rest.  The bucket walk then meets the clamped
particles among that bucket's, so the vorticity pass does in either
neighbour mode: bit-identical results."""
import itertools

import numpy as np
import pytest

import pbf_b200 as P
from pbf_b200 import scenes

pytestmark = pytest.mark.gpu

H = 0.1


def buckets(cells, mask):
    c = np.asarray(cells, np.int64)
    return ((c[..., 0] * 73856093) ^ (c[..., 1] * 19349663) ^ (c[..., 2] * 83492791)) & mask


def around(c, r):
    return np.asarray(c) + np.array(list(itertools.product(range(-r, r + 1), repeat=3)))


def colliding(hash_size, axis):
    """The first (c, M): c a cell at the lower wall of `axis` with no collision
    between its neighbours and the cells within two of it, M a cell beyond the
    wall, beside c along the wall, in the bucket of one of c's neighbours."""
    mask, along = hash_size - 1, [k for k in range(3) if k != axis]
    for u, v in itertools.product(range(2, 30), repeat=2):
        c = np.zeros(3, int)
        c[along] = u, v
        near, two = around(c, 1), around(c, 2)
        hn, ht = buckets(near, mask), buckets(two, mask)
        same = (near[:, None] == two[None]).all(-1)
        if ((hn[:, None] == ht[None]) & ~same).any():
            continue
        for m, du, dv in itertools.product((3, 4, 5), (-1, 0, 1), (-1, 0, 1)):
            M = c.copy()
            M[axis] = -m
            M[along] += du, dv
            if (hn == buckets(M, mask)).any():
                return [(hash_size, axis, tuple(map(int, c)), tuple(map(int, M)))]
    return []


CASES = [x for hs in (1 << 8, 1 << 9, 1 << 10, 1 << 11, 1 << 12, 1 << 13) for axis in range(3) for x in colliding(hs, axis)]
assert len(CASES) >= 10


@pytest.mark.parametrize("hash_size,axis,c,M", CASES)
def test_clamped_beside_resting_ones(have_gpu, hash_size, axis, c, M):
    rng = np.random.default_rng(2)
    dt = 1.0 / 60.0
    # both groups close to the point of the wall between the two cells' middles
    c, M, into = np.array(c), np.array(M), np.eye(3)[axis]
    mid = 0.5 * (c + M + 1.0) * H * (1.0 - into)
    lean = (M - c) * H * (1.0 - into)
    rest = mid - 0.15 * lean + 0.05 * into + rng.uniform(-0.01, 0.01, (12, 3))
    rest_v = rng.normal(size=(12, 3)) * 0.05
    land = mid + 0.15 * lean + rng.uniform(-0.01, 0.01, (12, 3)) * (1.0 - into)
    start = land + 0.04 * into
    target = land + ((M[axis] + 0.5) * H + rng.uniform(-0.01, 0.01, (12, 1))) * into  # the predicted place
    fast_v = (target - start) / dt
    pos = np.concatenate([rest, start]).astype(np.float32)
    vel = np.concatenate([rest_v, fast_v]).astype(np.float32)
    cells = np.floor((pos + vel * np.float32(dt)) / H)
    assert (cells[:12] == c).all() and (cells[12:] == M).all()
    cfg = scenes.base_config(H, H / 2, (3.2, 3.2, 3.2), 1, 2, dt, len(pos), hash_size)
    cfg.gravity[:] = [0.0, 0.0, 0.0]
    cfg.enable_scorr = 0
    cfg.cohesion_strength = 0.0
    cfg.rho0 = 1e5  # thin fluid: no density correction moves anybody
    cfg.vorticity_epsilon = 0.5
    out = []
    for mode in (4, 8):
        fl = P.PBFluids(cfg)
        fl.set_option(1, mode)
        b = P.Batch(cfg, [dict(n=len(pos), bounds_min=tuple(cfg.bounds_min), bounds_max=tuple(cfg.bounds_max),
                               hash_size=hash_size)] * 2)
        b.set_option(P.BOPT_NEIGHBOUR_MODE, mode)
        fl.setParticles(P.make_particles(pos, vel))
        for k in range(2):
            b.set_particles(k, P.make_particles(pos, vel))
        fl.step()
        b.step()
        out += [fl.readbackParticles(), b.read_particles(0), b.read_particles(1)]
    assert (out[0]["pos"][12:, axis] == 0.0).all()  # clamped at the wall
    for o in out[1:]:
        assert np.array_equal(out[0]["pos"], o["pos"]) and np.array_equal(out[0]["vel"], o["vel"])
