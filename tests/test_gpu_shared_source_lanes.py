"""In-ball source samples dealt out over a warp with several owners: per-walk values of a
launch whose warps are full (more than 16 warps' worth of walks on every SM) against the
same walks in a launch that gives each walk a warp of its own.

Both launches add the same samples of a ball in the same order, so the values agree to the
rounding of a different instruction selection: 64 terms of 2^-22 each on sums of the size
of the largest value, 2e-5 of it.  A sample dealt to the wrong owner, dropped or added
twice changes a value by its share of a ball's source, some 1e-2 of it."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def pure_samples(gpu, bvh, problem, pts, options):
    from n2w._lib import call

    n = len(pts) * options.walks_per_point
    p = gpu.DeviceBuffer.from_array(pts)
    val, steps, forced, ov = (gpu.DeviceBuffer(4 * n) for _ in range(4))
    call("n2w_wos_pure_samples", bvh.handle, C.byref(problem), p.ptr, len(pts), C.byref(options), val.ptr, steps.ptr,
         forced.ptr, ov.ptr, None)
    call("n2w_device_sync")
    assert not ov.download(np.int32).any()
    return val.download(np.float32), steps.download(np.int32)


@pytest.fixture(scope="module")
def bvh(gpu):
    m = gpu.Mesh.bumpy_sphere_trig(32, 64, 0.08, 6, 8)
    m.normalize()
    return gpu.Bvh(m, 4, "sah")


@pytest.mark.parametrize("samples", [4, 5, 16, 33, 64])
def test_full_warps_equal_single_walk_warps(gpu, bvh, samples):
    problem = gpu.problem_sinprod(3.0 * np.pi)
    problem.source_samples = samples
    pts = np.random.default_rng(samples).uniform(-0.4, 0.4, (4000, 3)).astype(np.float32)
    o = gpu.walk_options(walks_per_point=25, max_steps=64, epsilon=1e-3, seed=31 + samples)
    full, full_steps = pure_samples(gpu, bvh, problem, pts, o)  # 100,000 walks: 32 lanes a warp
    one, one_steps = pure_samples(gpu, bvh, problem, pts[:80], o)  # 2,000 walks: one lane a warp
    assert np.array_equal(full_steps[:len(one)], one_steps) and one_steps.max() > 3
    assert np.abs(full[:len(one)] - one).max() <= 2e-5 * np.abs(one).max()
    # the other walks, by their means: the same problem at the same points with other seeds
    o2 = gpu.walk_options(walks_per_point=25, max_steps=64, epsilon=1e-3, seed=77 + samples)
    again, _ = pure_samples(gpu, bvh, problem, pts, o2)
    sigma = np.sqrt((full.var() + again.var()) / len(full))
    assert abs(full.mean() - again.mean()) < 6 * sigma


def test_batches_with_one_sample_count(gpu, bvh):
    """Batches run full warps at any size: every instance's sums equal its solo run's."""
    scene = gpu.Scene([bvh])
    rng = np.random.default_rng(9)
    o = gpu.walk_options(max_steps=64, epsilon=1e-3)
    for samples in (4, 5, 16, 33, 64):
        problem = gpu.problem_sinprod(3.0 * np.pi)
        problem.source_samples = samples
        inst = [{"mesh": 0, "problem": 0, "points": rng.uniform(-0.4, 0.4, (9, 3)).astype(np.float32),
                 "walks_per_point": 30, "seed": 500 + i} for i in range(24)]
        b = gpu.Batch(scene, [problem], inst, o)
        b.launch()
        for i, (got, it) in enumerate(zip(b.results(), inst)):
            one = gpu.walk_options(walks_per_point=30, max_steps=64, epsilon=1e-3, seed=500 + i)
            want, _ = gpu.wos_estimate(bvh, problem, it["points"], options=one)
            assert np.array_equal(got["mean_steps"], want["mean_steps"])
            assert np.allclose(got["sum"], want["sum"], rtol=0, atol=2e-5 * 30 * np.abs(want["mean"]).max()), (samples, i)
