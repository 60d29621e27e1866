"""Closest-point queries of the same mesh at very small and very large scales.  Above
about 1e9 the products of a triangle test overflow for some triangles, which then have no
distance at all; the answer is the closest of the others, which a search must not have
ruled out on account of the ones that dropped out.  Against the counted query, which
searches the whole tree from its root."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-24, 1e-18, 1e-12, 1e-8, 1e-4, 1e4, 1e8, 1e10, 1e12, 1e17, 1e19])
@pytest.mark.parametrize("level", [2, 4])
def test_queries_at_scale(gpu, level, scale):
    v, t = gpu.Mesh.icosphere_displaced(level, 0.12, 3.0, 4, 0.5, 12345).arrays()
    s = np.float32(scale)
    bvh = gpu.Bvh(gpu.Mesh.from_arrays(v * s, t), 4, "sah")
    rng = np.random.default_rng(level)
    pts = np.concatenate([rng.uniform(-1.3, 1.3, (20_000, 3)),
                          v[rng.integers(0, len(v), 20_000)] * (1 + rng.normal(size=(20_000, 1)) * 1e-3)])
    pts = pts.astype(np.float32) * s
    want = bvh.query(pts, counted=True)
    for part in (slice(None), slice(0, 2000), slice(-2000, None)):  # a lane per query, a warp per query
        got = bvh.query(pts[part])
        assert not got["overflow"].any()
        for key in ("distance2", "closest"):
            assert np.array_equal(got[key].view(np.uint32), want[key][part].view(np.uint32)), key
        assert np.array_equal(got["triangle_id"], want["triangle_id"][part])


def test_walks_at_a_large_scale(gpu):
    """Walks inside a mesh whose triangle tests overflow in part: every step's search finds a triangle."""
    v, t = gpu.Mesh.icosphere_displaced(3, 0.12, 3.0, 4, 0.5, 12345).arrays()
    s = np.float32(1e12)
    bvh = gpu.Bvh(gpu.Mesh.from_arrays(v * s, t), 4, "sah")
    pts = np.random.default_rng(5).uniform(-0.3, 0.3, (64, 3)).astype(np.float32) * s
    o = gpu.walk_options(walks_per_point=64, max_steps=256, epsilon=1e-2 * float(s))
    r, c = gpu.wos_estimate(bvh, gpu.problem_charges_seeded(8, 1.6, 2.0, 1), pts, options=o)
    assert (r["count"] == 64).all() and c["overflow"] == 0
    # a query without a hit ends its walk where it is: at this epsilon walks take about a dozen steps
    assert r["mean_steps"].mean() > 5
