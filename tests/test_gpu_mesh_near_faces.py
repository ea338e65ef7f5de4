"""Nearest-face searches where rounding is as large as the distance: points a
few units in the last place off a mesh's vertices and faces.  A face's nearest
point is rounded at the size of its coordinates, so it can lie outside the
face's own box; every query still has a face, at the distance brute force in
64 bits finds, within FP32 rounding of the coordinates."""
import numpy as np
import pytest

import pbf_b200 as P
from pbf_b200 import scenes
from test_gpu_mesh_search import nearest

pytestmark = pytest.mark.gpu

TETRA = (np.array([[0.0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]]),
         np.array([[0, 2, 1], [0, 1, 3], [0, 3, 2], [1, 2, 3]], np.int32))
CUBE = (np.array([[x, y, z] for x in (0.0, 1) for y in (0.0, 1) for z in (0.0, 1)]),
        np.array([[0, 1, 3], [0, 3, 2], [4, 6, 7], [4, 7, 5], [0, 4, 5], [0, 5, 1], [2, 3, 7], [2, 7, 6], [0, 2, 6],
                  [0, 6, 4], [1, 5, 7], [1, 7, 3]], np.int32))
TRIANGLE = (np.array([[0.0, 0, 0], [1, 0, 0], [0.4, 0.8, 0]]), np.array([[0, 1, 2]], np.int32))
SHAPES = {"tetrahedron": TETRA, "cube": CUBE, "triangle": TRIANGLE}


def turned(v, rng):
    """v rotated at random, scaled and moved, as the mesh stores it (FP32)."""
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    return ((v - v.mean(0)) @ (q * np.sign(np.diag(r))).T * rng.uniform(0.5, 3.0)
            + rng.uniform(-1.0, 1.0, 3)).astype(np.float32)


def beside(v, n, ulps, rng):
    """n points up to `ulps` units in the last place off vertices."""
    at = v[rng.integers(0, len(v), n)]
    return (at + rng.integers(-ulps, ulps + 1, at.shape) * np.spacing(np.abs(at))).astype(np.float32)


def plane(n, z, rng):
    """A grid of quads at z, its heights one unit in the last place off."""
    x, y = np.meshgrid(np.arange(n + 1) / 16.0, np.arange(n + 1) / 16.0, indexing="ij")
    zz = np.float32(z) + rng.integers(-1, 2, x.shape) * np.spacing(np.float32(z))
    v = np.stack([x, y, zz], -1).reshape(-1, 3).astype(np.float32)
    c = (np.arange(n)[:, None] * (n + 1) + np.arange(n)).reshape(-1)
    f = np.concatenate([np.stack([c, c + n + 1, c + n + 2], 1), np.stack([c, c + n + 2, c + 1], 1)])
    return v, f.astype(np.int32)


def check(v, f, pts, face, point):
    d = np.concatenate([nearest(v.astype(np.float64)[f], p) for p in np.array_split(pts, 1 + len(pts) * len(f) // 200000)])
    tol = 4e-6 * (np.abs(pts).max() + np.ptp(v, axis=0).max())  # a few FP32 ulps of the coordinates
    assert (face >= 0).all(), f"{(face < 0).sum()} of {len(pts)} without a face"
    assert np.abs(np.linalg.norm(pts.astype(np.float64) - point, axis=1) - d.min(1)).max() <= tol
    assert (d[np.arange(len(pts)), face] <= d.min(1) + tol).all()


@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_queries_beside_vertices(have_gpu, shape):
    v0, f = SHAPES[shape]
    rng = np.random.default_rng(17)
    for _ in range(20):
        v = turned(v0, rng)
        sdf = P.SDFBoundary()
        sdf.buildFromMesh(v.astype(np.float64), f, float(np.ptp(v, axis=0).max()) / 4)
        pts = np.concatenate([beside(v, 1500, k, rng) for k in (1, 2, 3, 4)])
        check(v, f, pts, *sdf.closest_many(pts))


@pytest.mark.parametrize("z", [0.25, 0.5, 1.0])
@pytest.mark.parametrize("n", [1, 8, 40])
def test_queries_over_a_plane(have_gpu, z, n):
    """From 2 faces (all in the first round of a search) to 3,200."""
    rng = np.random.default_rng(5)
    v, f = plane(n, z, rng)
    sdf = P.SDFBoundary()
    sdf.buildFromMesh(v.astype(np.float64), f, n / 16.0 / 4)
    m = 20000 if n < 40 else 3000
    over = np.stack([rng.uniform(0, n / 16.0, m), rng.uniform(0, n / 16.0, m),
                     z + rng.choice([1e-7, 1e-5, 1e-3, 1e-2], m) * rng.normal(size=m)], 1).astype(np.float32)
    pts = np.concatenate([over, beside(v, m // 4, 3, rng)])
    check(v, f, pts, *sdf.closest_many(pts))


def test_grid_over_a_plane(have_gpu):
    """Voxels a few units in the last place off the plane's faces."""
    v, f = plane(8, 0.5, np.random.default_rng(6))
    v64 = v.astype(np.float64)
    sdf = P.SDFBoundary()
    sdf.buildFromMesh(v64, f, 1.0 / 32)
    dims, org, _ = sdf._info()
    ax = [np.float32(org[k] + np.arange(dims[k]) / 32) for k in range(3)]
    pts = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    d = np.concatenate([nearest(v64[f], p).min(1) for p in np.array_split(pts, 20)])
    assert np.abs(np.abs(sdf.distances()) - d).max() <= 4e-6 * (np.abs(pts).max() + 1.0)


@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_forces_beside_vertices(have_gpu, shape):
    """Every contact candidate pushes: each lies on the mesh within rounding."""
    v0, f = SHAPES[shape]
    rng = np.random.default_rng(23)
    for _ in range(10):
        v = turned(v0, rng)
        pts = np.concatenate([beside(v, 5000, k, rng) for k in (1, 2, 3, 4)])
        size = float(np.ptp(v, axis=0).max())
        sdf = P.SDFBoundary()
        sdf.buildFromMesh(v.astype(np.float64), f, size / 8)
        cfg = scenes.base_config(0.04, 0.02, (8.0, 8.0, 8.0), 1, 1, 1.0 / 60.0, len(pts))
        cfg.bounds_min[:] = [-8.0, -8.0, -8.0]
        fl = P.PBFluids(cfg)
        fl.setParticles(P.make_particles(pts, np.zeros_like(pts)))
        fl.setSDFBoundary(sdf)
        fl.setSDFPadding(0.0)
        fl.filterContactCandidates(size)
        assert len(fl.readbackContactCandidates()) == len(pts)
        force, contacts = fl.computeContactForces(size, False)
        assert contacts == len(pts) and np.isfinite(force).all()
