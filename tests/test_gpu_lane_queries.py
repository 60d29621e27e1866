"""Launches large enough for a lane per query, and their finisher: the meshes, point sets
and masks that other tests bring in counts that a warp per query answers.  Every output
equals the counted query's bit for bit, at ragged counts, and nothing past the end is
written."""
import numpy as np
import pytest

import oracle
from test_gpu_frames import _mesh, _points

pytestmark = pytest.mark.gpu

LANES = 32769  # one lane per query from here on, on every tree
GUARD = 0x7F7F7F7F


def guarded_query(gpu, bvh, pts, active=None):
    n = len(pts)
    p = gpu.DeviceBuffer.from_array(np.ascontiguousarray(pts, np.float32))
    out = {k: gpu.DeviceBuffer.from_array(np.full(w * (n + 8), GUARD, np.uint32)) for k, w in
           (("distance2", 1), ("closest", 3), ("triangle_id", 1), ("overflow", 1))}
    act = None if active is None else gpu.DeviceBuffer.from_array(active)
    bvh.query_device(p.ptr, n, out["distance2"].ptr, out["closest"].ptr, out["triangle_id"].ptr, out["overflow"].ptr,
                     d_active=None if act is None else act.ptr)
    got = {}
    for k, b in out.items():
        a, w = b.download(np.uint32), 3 if k == "closest" else 1
        assert (a[w * n:] == GUARD).all(), k
        got[k] = a[:w * n].reshape(n, w) if w > 1 else a[:n]
    return got


def check(gpu, bvh, pts, masked=False, seed=0):
    want = bvh.query(pts, counted=True)
    active = None
    if masked:
        active = (np.random.default_rng(seed).random(len(pts)) < 0.6).astype(np.uint8)
        off = active == 0
        want["distance2"][off], want["closest"][off] = 0.0, pts[off]
        want["triangle_id"][off] = -1
    got = guarded_query(gpu, bvh, pts, active)
    for k in ("distance2", "closest", "triangle_id"):
        assert np.array_equal(got[k], np.ascontiguousarray(want[k]).view(np.uint32)), k
    assert not got["overflow"].any()
    return want


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("n", [LANES, LANES + 37, 100_003])
@pytest.mark.parametrize("name", ["triangle", "plane", "soup", "ico0", "ico3", "ico6", "shifted"])
def test_meshes_and_points_of_the_framed_queries(gpu, name, n, masked):
    m = _mesh(gpu, name)
    v, _ = m.arrays()
    pts = _points(v, 2000)
    reps = -(-n // len(pts))
    check(gpu, gpu.Bvh(m, 4, "sah"), np.tile(pts, (reps, 1))[:n].copy(), masked, n)


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("n", [16_384, 16_385, 24_001, 32_768, LANES, 131_077])
def test_around_the_switches(gpu, n, masked):
    """The counts at which launches change from warps to lanes that keep the short queries, and to lanes that keep all,
    with points near and far from the surface, and very far ones."""
    m = gpu.Mesh.icosphere_displaced(5, 0.12, 3.0, 4, 0.5, 12345)
    v, t = m.arrays()
    rng = np.random.default_rng(n)
    tri = v[t[rng.integers(0, len(t), n)]]
    pts = (tri.mean(1) + rng.normal(size=(n, 3)) * np.exp(rng.uniform(-9, 1, (n, 1)))).astype(np.float32)
    pts[::977] *= 1e5
    check(gpu, gpu.Bvh(m, 4, "sah"), pts, masked, n)


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("n", [LANES + 37, 100_003])
def test_centre_of_a_closed_mesh(gpu, n, masked):
    """Far from the surface in every direction; a part against the brute force."""
    m = gpu.Mesh.bumpy_sphere_trig(128, 256, 0.08, 6, 8)
    m.normalize()
    v, t = m.arrays()
    rng = np.random.default_rng(n)
    pts = np.where(rng.random((n, 1)) < 0.5, rng.uniform(-0.25, 0.25, (n, 3)), rng.uniform(-1.2, 1.2, (n, 3)))
    pts = pts.astype(np.float32)
    want = check(gpu, gpu.Bvh(m, 4, "sah"), pts, masked, n)
    if not masked:
        bf = oracle.bruteforce(v, t, pts[-600:])
        assert np.array_equal(want["distance2"][-600:].view(np.uint32), bf["distance2"].view(np.uint32))
        assert np.array_equal(want["triangle_id"][-600:], bf["triangle_id"])


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("n", [LANES + 37, 70_001])
def test_queries_that_no_lane_may_finish(gpu, n, masked):
    """800 copies of one triangle over a sphere: every search that ends at them has to test all 800, for the lowest id,
    which is more than any lane's budget (112 over frames, 384 over boxes) at these counts: every third query is handed
    off to the finisher, the rest end within their lanes."""
    m = gpu.Mesh.icosphere_displaced(3, 0.12, 3.0, 4, 0.5, 12345)
    v, t = m.arrays()
    k = len(v)
    tri = np.array([[3.0, -0.2, -0.2], [3.0, 0.4, -0.2], [3.0, -0.2, 0.4]], np.float32)
    tris = np.concatenate([t, np.tile([[k, k + 1, k + 2]], (800, 1))])
    perm = np.random.default_rng(2).permutation(len(tris))
    bvh = gpu.Bvh(gpu.Mesh.from_arrays(np.concatenate([v, tri]), tris[perm]), 4, "sah")
    lowest = np.nonzero(perm >= len(t))[0].min()
    rng = np.random.default_rng(n)
    pts = v[rng.integers(0, k, n)] * (1 + rng.uniform(-0.01, 0.01, (n, 1)))
    pts[::3] = np.array([3.0, 0.0, 0.0]) + rng.uniform(-0.1, 0.1, (len(pts[::3]), 3))
    want = check(gpu, bvh, pts.astype(np.float32), masked, n)
    hit = want["triangle_id"][::3]
    assert set(np.unique(hit)) <= {-1, lowest} and (hit == lowest).any()
