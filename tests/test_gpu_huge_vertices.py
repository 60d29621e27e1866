"""Meshes with a vertex at infinity or near the end of the float range, as a broken file
or a far-field stand-in has: the triangles with finite distances are found all the same."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [1e19, 1e30, 1e36, 1e37, 3e38, np.inf])
@pytest.mark.parametrize("n", [500, 33_003])
def test_finite_triangles_beside_a_huge_one(gpu, far, n):
    v, t = gpu.Mesh.icosphere_displaced(3, 0.12, 3.0, 4, 0.5, 12345).arrays()
    f = np.float32(far)
    corners = np.array([[f, 0.3, 0.1], [0.0, -f, 2.0], [3.0, 3.0, 3.0], [3.0, 4.0, 3.0]], np.float32)
    k = len(v)
    mesh = gpu.Mesh.from_arrays(np.concatenate([v, corners]),
                                np.concatenate([t, [[k, k + 2, k + 3], [k + 1, k + 2, k + 3]]]))
    verts, tris = mesh.arrays()
    bvh = gpu.Bvh(mesh, 4, "sah")
    rng = np.random.default_rng(1)
    pts = np.concatenate([rng.uniform(-1.3, 1.3, (n - 100, 3)),
                          v[rng.integers(0, k, 100)] * (1 + rng.uniform(-1e-3, 1e-3, (100, 1)))]).astype(np.float32)
    want = bvh.query(pts, counted=True)
    with np.errstate(all="ignore"):
        bf = oracle.bruteforce(verts, tris, pts[-500:])
    assert np.array_equal(want["triangle_id"][-500:], bf["triangle_id"])
    got = bvh.query(pts)
    assert not got["overflow"].any()
    for key in ("distance2", "closest"):
        assert np.array_equal(got[key].view(np.uint32), want[key].view(np.uint32)), key
    assert np.array_equal(got["triangle_id"], want["triangle_id"])
