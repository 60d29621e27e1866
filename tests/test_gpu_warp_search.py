"""Warp-per-query launches (small query counts) against the counted query, at the
sizes around the warp, the block and the switch to one lane per query."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SWITCH = 32768  # launches above this run one lane per query


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, SWITCH - 1, SWITCH, SWITCH + 1])
def test_small_launches_equal_counted_query(gpu, n, masked):
    m = gpu.Mesh.icosphere_displaced(4, 0.12, 3.0, 4, 0.5, 12345)
    bvh = gpu.Bvh(m, 4, "sah")
    rng = np.random.default_rng(n)
    pts = rng.uniform(-1.4, 1.4, (n, 3)).astype(np.float32)
    pts[0] = 0.0  # far from the surface in every direction
    if n > 2:
        pts[1], pts[2] = (np.nan, 0.0, 0.0), (1e4, -1e4, 0.0)
    want = bvh.query(pts, counted=True)
    active = (rng.random(n) < 0.5).astype(np.uint8) if masked else None
    got = bvh.query(pts, active=active)
    if masked:
        off = active == 0
        want["distance2"][off], want["closest"][off] = 0.0, pts[off]
        want["triangle_id"][off], want["overflow"][off] = -1, 0
    for k in ("distance2", "closest"):
        assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), k
    for k in ("triangle_id", "overflow"):
        assert np.array_equal(got[k], want[k]), k
