"""Closest-point traversals over the framed nodes against the counted query,
which runs the same arithmetic over the axis-aligned nodes (pinned to the CPU
restatement elsewhere): every output equal bit for bit, whatever the mesh's
size, shape and position and wherever the points lie."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(gpu, name):
    rng = np.random.default_rng(5)
    if name == "triangle":
        return gpu.Mesh.from_arrays([[0, 0, 0], [1, 0, 0], [0, 1, 0.5]], [[0, 1, 2]])
    if name == "plane":  # coplanar grid: every patch is flat, exact ties along edges
        g = np.arange(33, dtype=np.float32) / 16 - 1
        v = np.stack(np.meshgrid(g, g, [0.25], indexing="ij"), -1).reshape(-1, 3)
        i = np.arange(32)[:, None] * 33 + np.arange(32)
        t = np.concatenate([np.stack([i, i + 33, i + 1], -1), np.stack([i + 1, i + 33, i + 34], -1)]).reshape(-1, 3)
        return gpu.Mesh.from_arrays(v, t)
    if name == "soup":  # random triangles of very uneven sizes, some degenerate, some twice
        c = rng.normal(size=(3000, 1, 3))
        v = (c + rng.normal(size=(3000, 3, 3)) * np.exp(rng.uniform(-8, 0, (3000, 1, 1)))).astype(np.float32)
        v[::50, 2] = v[::50, 1]
        v[1::50] = v[::50]
        return gpu.Mesh.from_arrays(v.reshape(-1, 3), np.arange(9000).reshape(-1, 3))
    level = {"ico0": 0, "ico3": 3, "ico6": 6, "shifted": 4}[name]
    m = gpu.Mesh.icosphere_displaced(level, 0.12, 3.0, 4, 0.5, 12345)
    if name == "shifted":  # coordinates a hundred times the extent
        v, t = m.arrays()
        m = gpu.Mesh.from_arrays(v + np.float32([100, -70, 30]), t)
    return m


def _points(v, n):
    rng = np.random.default_rng(9)
    lo, hi = v.min(0), v.max(0)
    c, e = (lo + hi) / 2, (hi - lo).max()
    near = v[rng.integers(0, len(v), n)] + rng.normal(size=(n, 3)) * e * np.exp(rng.uniform(-14, -1, (n, 1)))
    far = c + rng.normal(size=(n, 3)) * e * np.exp(rng.uniform(0, 12, (n, 1)))
    box = rng.uniform(c - 0.7 * e, c + 0.7 * e, (n, 3))
    odd = np.array([c, lo, hi, [np.inf, 0, 0], [np.nan, 0, 0], [1e19, 0, 0], [3e38, 3e38, 3e38], v[0]])
    return np.concatenate([near, far, box, odd, c + (v[:n] - c) * 1e-6]).astype(np.float32)


@pytest.mark.parametrize("method,leaf", [("sah", 4), ("spatial_median", 8)])
@pytest.mark.parametrize("name", ["triangle", "plane", "soup", "ico0", "ico3", "ico6", "shifted"])
def test_framed_query_equals_counted_query(gpu, name, method, leaf):
    m = _mesh(gpu, name)
    v, _ = m.arrays()
    bvh = gpu.Bvh(m, leaf, method)
    pts = _points(v, 2000)
    want = bvh.query(pts, counted=True)
    got = bvh.query(pts)
    assert not want["overflow"].any() and not got["overflow"].any()
    for k in ("distance2", "closest"):
        assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), k
    assert np.array_equal(got["triangle_id"], want["triangle_id"])
