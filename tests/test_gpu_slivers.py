"""Soups of slivers, triangles whose computed closest points are off by more than a seed
cell's size: a search must not leave out what only the exact distances rule out.  Against
the counted query, which searches the whole tree from its root."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,width", [(4, 1e-6), (13, 1e-8), (5, 1e-6), (5, 1e-8), (6, 1e-4), (7, 1e-2)])
def test_sliver_soup(gpu, seed, width):
    n, length = 3000, 0.5
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1, 1, (n, 1, 3))
    d, e = rng.normal(size=(n, 3)), None
    d /= np.linalg.norm(d, axis=1)[:, None]
    e = rng.normal(size=(n, 3))
    e /= np.linalg.norm(e, axis=1)[:, None]
    a = c[:, 0]
    v = np.stack([a, a + d * length, a + d * length * rng.uniform(-0.5, 1.5, (n, 1)) + e * width], 1)
    bvh = gpu.Bvh(gpu.Mesh.from_arrays(v.reshape(-1, 3).astype(np.float32), np.arange(3 * n).reshape(-1, 3)), 4, "sah")
    pts = np.concatenate([rng.uniform(-1.2, 1.2, (20_000, 3)),
                          v[rng.integers(0, n, 20_000)].mean(1) +
                          rng.normal(size=(20_000, 3)) * 10.0 ** rng.uniform(-6, -1, (20_000, 1))]).astype(np.float32)
    want = bvh.query(pts, counted=True)
    parts = [slice(None)] + [slice(i, i + 4000) for i in range(0, 40_000, 4000)]  # a lane, then a warp per query
    for part in parts:
        got = bvh.query(pts[part])
        for key in ("distance2", "closest"):
            assert np.array_equal(got[key].view(np.uint32), want[key][part].view(np.uint32)), key
        assert np.array_equal(got["triangle_id"], want["triangle_id"][part])
