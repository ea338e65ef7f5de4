"""Nearest-face searches (k_mesh.cu, a warp per search) against brute force in
64 bits: distances within FP32 rounding of the coordinates' size, the face
returned among the nearest, for meshes from one face to more than a warp can
list, points on vertices and edges, inside, far away and not finite."""
import numpy as np
import pytest

import pbf_b200 as P
from pbf_b200 import scenes
from test_gpu_scenes import grid_cube

pytestmark = pytest.mark.gpu


def nearest(tri, pts):
    """Distance of every point to every face (points x faces), FP64."""
    a, b, c = (tri[None, :, k] for k in range(3))
    p = pts[:, None].astype(np.float64)
    ab, ac, bc = b - a, c - a, c - b

    def dot(x, y):
        return (x * y).sum(-1, keepdims=True)

    def edge(start, e):
        return start + e * np.clip(dot(p - start, e) / dot(e, e), 0.0, 1.0)

    n = np.cross(ab, ac)
    flat = p - n * (dot(p - a, n) / dot(n, n))
    inside = ((dot(np.cross(ab, flat - a), n) >= 0) & (dot(np.cross(bc, flat - b), n) >= 0)
              & (dot(np.cross(-ac, flat - c), n) >= 0))
    d = [np.linalg.norm(p - q, axis=-1) for q in (edge(a, ab), edge(a, ac), edge(b, bc))]
    d.append(np.where(inside[..., 0], np.linalg.norm(p - flat, axis=-1), np.inf))
    return np.min(d, axis=0)


MESHES = {
    "one": lambda: (np.array([[0.0, 0, 0], [1, 0, 0], [0, 1, 0]]), np.array([[0, 1, 2]], np.int32)),
    "two": lambda: (np.array([[0.0, 0, 0], [1, 0, 0], [0, 1, 0], [1, 1, 0]]), np.array([[0, 1, 2], [2, 1, 3]], np.int32)),
    "33": lambda: (lambda v, f: (v, f[:33]))(*scenes.icosphere(1, 0.3, (0.1, 0.2, 0.3))),
    "320": lambda: scenes.icosphere(2, 0.2, (0.8, 0.3, 0.5)),
    "cube": lambda: grid_cube(8),
    # one place many times over: all faces equally near
    "same": lambda: (np.tile([[0.0, 0, 0], [1, 0, 0], [0, 1, 0]], (100, 1)), np.arange(300, dtype=np.int32).reshape(-1, 3)),
}


@pytest.mark.parametrize("name", sorted(MESHES))
def test_queries_against_brute_force(have_gpu, name):
    v, f = MESHES[name]()
    tri = np.asarray(v, np.float32).astype(np.float64)[f]
    rng = np.random.default_rng(3)
    size = np.ptp(np.asarray(v), axis=0).max()
    lo, hi = np.min(v, 0) - 0.5 * size, np.max(v, 0) + 0.5 * size
    pts = np.concatenate([rng.uniform(lo, hi, (1500, 3)), np.asarray(v)[:200], (tri[:200, 0] + tri[:200, 1]) / 2,
                          np.mean(v, 0)[None], hi[None] + 50 * size]).astype(np.float32)
    sdf = P.SDFBoundary()
    sdf.buildFromMesh(v, f, size / 10)
    face, point = sdf.closest_many(pts)
    d = nearest(tri, pts)
    tol = 4e-6 * (np.abs(pts).max() + size)  # a few FP32 ulps of the coordinates
    got = np.linalg.norm(pts - point, axis=1)
    assert (face >= 0).all()
    assert np.abs(got - d.min(1)).max() <= tol
    assert (d[np.arange(len(pts)), face] <= d.min(1) + tol).all()


@pytest.mark.parametrize("name", ["320", "cube"])
def test_grid_against_brute_force(have_gpu, name):
    """Every voxel, those on the mesh's planes and corners among them."""
    v, f = MESHES[name]()
    sdf = P.SDFBoundary()
    cell = np.ptp(v, axis=0).max() / 12
    sdf.buildFromMesh(v, f, cell)
    dims, org, _ = sdf._info()
    ax = [np.float32(org[k] + np.arange(dims[k]) * cell) for k in range(3)]
    pts = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    tri = np.asarray(v, np.float32).astype(np.float64)[f]
    d = np.concatenate([nearest(tri, p).min(1) for p in np.array_split(pts, 20)])
    assert np.abs(np.abs(sdf.distances()) - d).max() <= 4e-6 * (np.abs(pts).max() + 1.0)


def test_more_waiting_nodes_than_fit(have_gpu):
    """Near the middle of a fine sphere every face is within the bound."""
    v, f = scenes.icosphere(6, 1.0, (0.0, 0.0, 0.0))
    sdf = P.SDFBoundary()
    sdf.buildFromMesh(v, f, 0.5)
    pts = (np.random.default_rng(1).normal(size=(40, 3)) * 1e-3).astype(np.float32)
    face, point = sdf.closest_many(pts)
    tri = np.asarray(v, np.float32).astype(np.float64)[f]
    d = np.stack([nearest(tri, p[None])[0] for p in pts])
    assert np.abs(np.linalg.norm(pts - point, axis=1) - d.min(1)).max() <= 4e-6
    assert (d[np.arange(len(pts)), face] <= d.min(1) + 4e-6).all()


def test_points_that_are_none(have_gpu):
    v, f = scenes.icosphere(2, 0.2, (0.8, 0.3, 0.5))
    sdf = P.SDFBoundary()
    sdf.buildFromMesh(v, f, 0.05)
    bad = np.array([[np.nan, 0, 0], [np.inf, 0, 0], [0, -np.inf, 0], [1e30, 0, 0]], np.float32)
    face, point = sdf.closest_many(bad)
    assert (face == -1).all() and (point == 0).all()


def test_queries_of_several_threads(have_gpu):
    """One SDF asked by four threads at once, with different numbers of points."""
    from concurrent.futures import ThreadPoolExecutor
    v, f = scenes.icosphere(3, 0.2, (0.8, 0.3, 0.5))
    sdf = P.SDFBoundary()
    sdf.buildFromMesh(v, f, 0.02)
    pts = np.random.default_rng(5).uniform(0.2, 1.2, (6000, 3)).astype(np.float32)
    face, point = sdf.closest_many(pts)
    d = sdf.sample(pts)
    with ThreadPoolExecutor(4) as ex:
        for n, (a, b, c) in ex.map(lambda n: (n, (*sdf.closest_many(pts[:n]), sdf.sample(pts[:n]))),
                                   [6000, 17, 3001, 1, 5999, 250] * 4):
            assert np.array_equal(a, face[:n]) and np.array_equal(b, point[:n]) and np.array_equal(c, d[:n])
