"""Launches that must not cost more than comparable ones: device times of pairs of
calls on one GPU, medians of interleaved runs, with wide bounds."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def timed_in_turn(gpu, calls, repeat=9):
    """Median device milliseconds of each call, run in turn."""
    stream, timer = gpu.Stream(), gpu.Timer()
    ms = [[] for _ in calls]
    for r in range(repeat + 2):
        for c, out in zip(calls, ms):
            timer.start(stream)
            c(stream)
            timer.stop(stream)
            t = timer.ms()
            if r >= 2:  # two rounds of warm-up
                out.append(t)
    return [float(np.median(x)) for x in ms]


def query_call(gpu, bvh, pts):
    n = len(pts)
    b = gpu.DeviceBuffer
    p, d2, cp, ids, ov = b.from_array(pts), b(4 * n), b(12 * n), b(4 * n), b(4 * n)
    return lambda s: bvh.query_device(p.ptr, n, d2.ptr, cp.ptr, ids.ptr, ov.ptr, 128, s)


def walk_call(gpu, bvh, pts, **options):
    from n2w._lib import call

    n = len(pts)
    p, st = gpu.DeviceBuffer.from_array(pts), gpu.PointStatsBuffers.allocate(n)
    o = gpu.walk_options(max_steps=256, epsilon=1e-3, **options)
    pb = gpu.problem_charges_seeded(8, 1.6, 2.0, 12345)
    return lambda s: call("n2w_wos_estimate", bvh.handle, C.byref(pb), p.ptr, n, C.byref(o), st.struct(), None, None,
                          s.handle)


def icosphere(gpu, level):
    m = gpu.Mesh.icosphere_displaced(level, 0.12, 3.0, 4, 0.5, 12345)
    m.normalize()
    return gpu.Bvh(m, 4, "sah")


@pytest.fixture(scope="module")
def small_and_large(gpu):
    return icosphere(gpu, 1), icosphere(gpu, 6)


def test_small_trees_stay_in_l1(gpu, small_and_large):
    """80 triangles (7 KB of nodes and triangles) against 81,920: the same queries take much less, the same walks too."""
    rng = np.random.default_rng(2)
    pts = rng.uniform(-1.2, 1.2, (1_000_003, 3)).astype(np.float32)
    small, large = timed_in_turn(gpu, [query_call(gpu, b, pts) for b in small_and_large])
    assert small < 0.65 * large, (small, large)
    pts = rng.uniform(-0.3, 0.3, (20_000, 3)).astype(np.float32)
    small, large = timed_in_turn(gpu, [walk_call(gpu, b, pts, walks_per_point=128) for b in small_and_large], 5)
    assert small < 0.65 * large, (small, large)


def test_short_queries_in_small_launches(gpu, small_and_large):
    """Queries close to the surface are short: 32,768 of them, the last size of the small launches' rules, take no more
    than 1.6 times what one query more takes."""
    m = gpu.Mesh.icosphere_displaced(6, 0.12, 3.0, 4, 0.5, 12345)
    m.normalize()
    v, t = m.arrays()
    rng = np.random.default_rng(3)
    tri = v[t[rng.integers(0, len(t), 32769)]]
    pts = (tri.mean(1) + rng.normal(size=(32769, 3)) * 3e-4).astype(np.float32)
    small, large = timed_in_turn(gpu, [query_call(gpu, small_and_large[1], p) for p in (pts[:-1], pts)])
    assert small < 1.6 * large, (small, large)


def test_few_walks_share_the_warps_that_the_caller_leaves(gpu, small_and_large):
    """150 x 16 walks in one warp per SM, half as many lanes as it has, take no more than twice what they take with the
    default launch shape, where each has a warp of its own."""
    pts = np.random.default_rng(4).uniform(-0.3, 0.3, (150, 3)).astype(np.float32)
    limited, free = timed_in_turn(gpu, [walk_call(gpu, small_and_large[1], pts, walks_per_point=16, **o) for o in
                                        (dict(blocks_per_sm=1, block_size=32), {})])
    assert limited < 2.0 * free, (limited, free)


def test_chunks_do_not_slow_small_batches(gpu, small_and_large):
    """A batch of few walks with the autotuner's smallest and largest chunks, and autotuned, against the batch as
    created: the chunk is a limit, and a lane's share of this launch is below one walk."""
    scene = gpu.Scene([small_and_large[1]])
    rng = np.random.default_rng(6)
    inst = [{"mesh": 0, "problem": 0, "points": rng.uniform(-0.3, 0.3, (100, 3)).astype(np.float32),
             "walks_per_point": 24, "seed": 40 + i} for i in range(4)]
    problems = [gpu.problem_charges_seeded(8, 1.6, 2.0, 3)]
    batches = [gpu.Batch(scene, problems, inst, gpu.walk_options(epsilon=1e-3)) for _ in range(4)]
    shape = {"block_size": 128, "blocks_per_sm": 0, "regen_threshold": 16, "reg_variant": batches[0].info()["reg_variant"]}
    batches[1].set_tuning({**shape, "chunk": 2})
    batches[2].set_tuning({**shape, "chunk": 16})
    batches[3].autotune(1.0)
    plain, two, sixteen, tuned = timed_in_turn(gpu, [lambda s, b=b: b.launch(s) for b in batches])
    assert max(two, sixteen, tuned) < 1.2 * plain, (plain, two, sixteen, tuned)
