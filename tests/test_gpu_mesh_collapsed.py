"""Meshes with collapsed faces: a face with two vertices in one place has no
nearest point where a query projects inside its remaining edge (0 / 0).
Searches pass such a face over."""
import numpy as np
import pytest

import pbf_b200 as P
from test_gpu_mesh_search import nearest
from test_gpu_scenes import grid_cube

pytestmark = pytest.mark.gpu


def test_grid_of_a_mesh_with_collapsed_faces(have_gpu):
    """A closed cube with a face along every edge that has no area."""
    v, f = grid_cube(4)
    v = np.asarray(v, np.float64)
    sdf = P.SDFBoundary()
    cell = 0.04
    sdf.buildFromMesh(v, np.concatenate([f, f[:, [0, 0, 1]], f[:, [1, 1, 2]], f[:, [2, 2, 0]]]), cell)
    dims, org, _ = sdf._info()
    ax = [np.float32(org[k] + np.arange(dims[k]) * cell) for k in range(3)]
    pts = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    d = np.concatenate([nearest(v[f], p).min(1) for p in np.array_split(pts, 40)])
    assert np.abs(np.abs(sdf.distances()) - d).max() <= 4e-6 * (np.abs(pts).max() + 1.0)


def test_one_whole_face_among_collapsed_ones(have_gpu):
    """Most searches look at collapsed faces alone before they meet the one
    that has a nearest point."""
    n = 200
    rng = np.random.default_rng(8)
    a = np.stack([np.arange(n) / 16.0, np.zeros(n), rng.uniform(-0.05, 0.05, n)], 1)
    collapsed = np.stack([a, a, a + [0.0, 0.1, 0.0]], 1)  # a point and an edge along y
    k = 83
    whole = collapsed[k] + [[0.0, 0.0, -0.01], [0.02, 0.0, -0.01], [0.0, 0.0, -0.01]]
    v = np.concatenate([collapsed.reshape(-1, 3), whole])
    f = np.arange(len(v), dtype=np.int32).reshape(-1, 3)
    sdf = P.SDFBoundary()
    sdf.buildFromMesh(v, f, 0.5)
    pts = np.stack([rng.uniform(0, a[-1, 0], 2000), rng.uniform(0.03, 0.07, 2000), rng.uniform(-0.2, 0.2, 2000)], 1)
    pts = pts.astype(np.float32)
    face, point = sdf.closest_many(pts)
    d = nearest(whole[None].astype(np.float32).astype(np.float64), pts)[:, 0]
    assert (face == n).all()
    assert np.abs(np.linalg.norm(pts - point, axis=1) - d).max() <= 4e-6 * (np.abs(pts).max() + 1.0)
