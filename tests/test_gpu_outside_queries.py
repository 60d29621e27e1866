"""Closest-point searches from points outside the seed grid's lattice (the mesh box
grown by 20 %): the answers of the counted query, for a bounded share of its work.

The counted query searches axis-aligned boxes; a plain estimate whose epsilon is
larger than any distance runs nothing but the points' first queries, and its run
counters are their node expansions and triangle tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SWITCH = 32768  # launches above this many points search with one lane per point


def sphere_points(v, n, extents, seed):
    """Points on the sphere around the mesh's box centre, `extents` times its largest extent away."""
    rng = np.random.default_rng(seed)
    lo, hi = v.min(0).astype(float), v.max(0).astype(float)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    return ((lo + hi) / 2 + d * (hi - lo).max() * extents).astype(np.float32)


def first_query_work(gpu, bvh, pts):
    """(nodes + triangles of the first queries) per point."""
    o = gpu.walk_options(walks_per_point=1, max_steps=1, epsilon=1e30)
    _, c = gpu.wos_estimate(bvh, gpu.problem_charges_seeded(8, 1.6, 2.0, 1), pts, options=o)
    assert c["steps"] == 0 and c["overflow"] == 0
    return (c["node_visits"] + c["tri_tests"]) / len(pts)


def assert_same_answers(got, want):
    for k in ("distance2", "closest"):
        assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), k
    assert np.array_equal(got["triangle_id"], want["triangle_id"])
    assert not got["overflow"].any()


@pytest.fixture(scope="module")
def sphere(gpu):
    m = gpu.Mesh.icosphere_displaced(5, 0.12, 3.0, 4, 0.5, 12345)
    return gpu.Bvh(m, 4, "sah"), m.arrays()[0]


@pytest.mark.parametrize("extents", [1.5, 5.0])
def test_seeds_outside_the_lattice(gpu, sphere, extents):
    """The seed lies in the direction of the point, so the search does half of the counted query's work or less."""
    bvh, v = sphere
    pts = sphere_points(v, SWITCH + 37, extents, 3)
    want = bvh.query(pts, counted=True)
    assert_same_answers(bvh.query(pts), want)
    assert_same_answers(bvh.query(pts[:1000]), {k: x[:1000] for k, x in want.items()})
    counted = (want["node_visits"] + want["tri_tests"]).mean()
    assert first_query_work(gpu, bvh, pts) < 0.5 * counted


def _patch(n, corner, eu, ev):
    """An n x n grid of quads, two triangles each."""
    g = np.linspace(0.0, 1.0, n + 1)
    u, w = (x.reshape(-1, 1) for x in np.meshgrid(g, g, indexing="ij"))
    v = np.asarray(corner, float) + u * np.asarray(eu, float) + w * np.asarray(ev, float)
    i = (np.arange(n)[:, None] * (n + 1) + np.arange(n)).ravel()
    return v, np.concatenate([np.stack([i, i + n + 1, i + 1], -1), np.stack([i + 1, i + n + 1, i + n + 2], -1)])


def _join(parts):
    off = np.cumsum([0] + [len(v) for v, _ in parts])
    return np.concatenate([v for v, _ in parts]).astype(np.float32), np.concatenate([t + o for (_, t), o in zip(parts, off)])


@pytest.fixture(scope="module")
def cube(gpu):
    """An axis-aligned cube, sides of 60 x 60 quads."""
    n, e = 60, 2 * np.eye(3)
    v, t = _join([_patch(n, -np.ones(3) + side * e[a], e[(a + 1) % 3], e[(a + 2) % 3]) for a in range(3) for side in (0, 1)])
    return gpu.Bvh(gpu.Mesh.from_arrays(v, t), 4, "sah"), v


def test_nearest_children_first(gpu, cube):
    """Flat sides seen from outside: many triangles lie within the seed's distance, few within the answer's."""
    bvh, v = cube
    pts = sphere_points(v, SWITCH + 37, 1.5, 4)
    want = bvh.query(pts, counted=True)
    assert_same_answers(bvh.query(pts), want)
    counted = (want["node_visits"] + want["tri_tests"]).mean()
    assert first_query_work(gpu, bvh, pts) < 4.0 * counted


@pytest.fixture(scope="module")
def needles(gpu):
    """The side of a cylinder in 2 x 5,000 triangles, each 2 long and 0.001 wide."""
    k = 5000
    a = np.arange(k) * 2 * np.pi / k
    lo = np.stack([np.cos(a), np.sin(a), -np.ones(k)], -1)
    i, j = np.arange(k), (np.arange(k) + 1) % k
    t = np.concatenate([np.stack([i, j, i + k], -1), np.stack([j, j + k, i + k], -1)])
    v = np.concatenate([lo, lo + [0, 0, 2]]).astype(np.float32)
    return gpu.Bvh(gpu.Mesh.from_arrays(v, t), 4, "sah"), v


@pytest.mark.parametrize("n", [1000, SWITCH + 37])
@pytest.mark.parametrize("where", ["inside", "outside"])
@pytest.mark.parametrize("name", ["cube", "needles"])
def test_trees_whose_frames_do_not_pay(gpu, request, name, where, n):
    """Axis-aligned sides and bundles of needles: the queries search the axis-aligned boxes, from seeds at least as
    good as the counted query's, so a lane does no more work than that."""
    bvh, v = request.getfixturevalue(name)
    pts = np.random.default_rng(6).uniform(-1.2, 1.2, (n, 3)).astype(np.float32) if where == "inside" else \
        sphere_points(v, n, 1.5, 6)
    want = bvh.query(pts, counted=True)
    assert_same_answers(bvh.query(pts), want)
    if n > SWITCH:
        assert first_query_work(gpu, bvh, pts) <= 1.0 * (want["node_visits"] + want["tri_tests"]).mean()


@pytest.mark.parametrize("extents,offset", [(5e3, 0.0), (5e4, 0.0), (0.5, 2e4), (50.0, 1e3)])
def test_far_coordinates_search_the_boxes(gpu, sphere, extents, offset):
    """Thousands of extents away, or with the mesh that far from the origin, the framed nodes' rounding margin covers
    whole patches; the search then does no more work than the counted query."""
    bvh, v = sphere
    if offset:
        _, t = gpu.Mesh.icosphere_displaced(5, 0.12, 3.0, 4, 0.5, 12345).arrays()
        v = v + np.float32(offset)
        bvh = gpu.Bvh(gpu.Mesh.from_arrays(v, t), 4, "sah")
    pts = sphere_points(v, SWITCH + 37, extents, 5)
    want = bvh.query(pts, counted=True)
    assert_same_answers(bvh.query(pts), want)
    assert_same_answers(bvh.query(pts[:1000]), {k: x[:1000] for k, x in want.items()})
    counted = (want["node_visits"] + want["tri_tests"]).mean()
    assert first_query_work(gpu, bvh, pts) <= 1.0 * counted


def test_few_far_points_among_near_ones(gpu, sphere):
    """Far points scattered through a launch of near ones, and whole warps of them: handed off at once, the rest not."""
    bvh, v = sphere
    rng = np.random.default_rng(8)
    pts = rng.uniform(-1.2, 1.2, (SWITCH + 37, 3)).astype(np.float32)
    far = sphere_points(v, len(pts), 5e3, 9)
    sel = np.zeros(len(pts), bool)
    sel[::41] = True  # less than one a warp
    sel[10_000:10_000 + 100] = True  # whole warps, from the middle of one
    sel[-3:] = True
    pts[sel] = far[sel]
    want = bvh.query(pts, counted=True)
    assert_same_answers(bvh.query(pts), want)
