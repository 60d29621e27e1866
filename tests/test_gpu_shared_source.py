"""In-ball source samples shared by a warp: walks of instances with different sample
counts, mixed in one launch (the lanes of a warp disagree, so each lane draws its
own), against each instance alone (its lanes agree and share them)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_shared_samples_equal_own_samples(gpu):
    m = gpu.Mesh.bumpy_sphere_trig(32, 64, 0.08, 6, 8)
    m.normalize()
    bvh = gpu.Bvh(m, 4, "sah")
    counts = [4, 5, 1, 16, 33, 64, 3, 7]  # around the threshold, dividing 32 or not, the largest
    problems = []
    for k in counts:
        p = gpu.problem_sinprod(3.0 * np.pi)
        p.source_samples = k
        problems.append(p)
    problems.append(gpu.problem_charges_seeded(8, 1.6, 2.0, 3))  # no source at all
    rng = np.random.default_rng(4)
    o = gpu.walk_options(max_steps=64, epsilon=1e-3)
    inst = [{"mesh": 0, "problem": i % len(problems), "points": rng.uniform(-0.4, 0.4, (1, 3)).astype(np.float32),
             "walks_per_point": 5, "seed": 100 + i} for i in range(40 * len(problems))]
    b = gpu.Batch(gpu.Scene([bvh]), problems, inst, o)
    b.launch()
    got = b.results()
    for i, (g, it) in enumerate(zip(got, inst)):
        one = gpu.walk_options(walks_per_point=5, max_steps=64, epsilon=1e-3, seed=100 + i)
        want, _ = gpu.wos_estimate(bvh, problems[it["problem"]], it["points"], options=one)
        assert np.array_equal(g["mean_steps"], want["mean_steps"]) and np.array_equal(g["count"], want["count"])
        # the same FP32 values summed in FP64 in another order
        assert np.allclose(g["sum"], want["sum"], rtol=1e-13, atol=1e-13 * 5 * 100), (i, counts)
