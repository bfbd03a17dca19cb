"""The group walk's classes of children (far, plain, odd) at the sizes and layouts where a wrong
class would show: groups of one point to several, coordinates shared by many points (d3 jiggles a
zero component), points nearer than distanceMin, chains of one-child cells, and a distanceMax that
cuts through a group. The walk of one point per warp makes the same traversal with every test on
every child, so the counters must agree exactly and the velocities up to the order of FP32 sums."""
import numpy as np
import pytest

from forcegpu._lib import (Q_WALK_APPLIES, Q_WALK_OPENS, Q_WALK_USEFUL, TUNE_WALK_GROUP, Engine,
                           desc_from_gpu)

pytestmark = pytest.mark.gpu


def points(kind, n, dims):
    rng = np.random.default_rng(n + dims)
    if kind == "grid":        # integer coordinates: most children share a coordinate
        x = rng.integers(-9, 10, (n, dims)).astype(np.float64)
    elif kind == "plane":     # one axis the same for every point, 0 and -0 mixed
        x = rng.normal(0, 100, (n, dims))
        x[:, -1] = np.where(np.arange(n) % 2 == 0, 0.0, -0.0)
    elif kind == "pairs":     # close pairs far apart: long chains, distanceMin
        x = np.repeat(rng.normal(0, 1000, ((n + 1) // 2, dims)), 2, axis=0)[:n]
        x = x + rng.normal(0, 0.4, (n, dims))
    else:                     # "cloud"
        x = rng.normal(0, 4 * n ** (1 / dims), (n, dims))
    pos4 = np.zeros((n, 4), np.float32)
    pos4[:, :dims] = x
    return pos4


def walk(pos4, dims, group, dmin2, dmax2):
    n = len(pos4)
    e = Engine(0)
    e.set_nodes(pos4, dims)
    e.set_forces([desc_from_gpu({"type": "manyBody", "version": 1, "strengths": np.full(n, -30.0),
                                 "distanceMin2": dmin2, "distanceMax2": dmax2, "theta2": 0.81}, 1, n)])
    e.set_seed(3)
    e.set_tuning(TUNE_WALK_GROUP, group)
    e.profile(2)
    e.enqueue(np.array([0.7]), 0.6)
    _, vel = e.sync()
    counts = [e.query(q) for q in (Q_WALK_USEFUL, Q_WALK_OPENS, Q_WALK_APPLIES)]
    e.close()
    return vel[:, :dims].astype(np.float64), counts


@pytest.mark.parametrize("kind", ["cloud", "grid", "plane", "pairs"])
@pytest.mark.parametrize("n,dims", [(2, 3), (31, 2), (33, 3), (65, 1), (4099, 3), (3001, 2)])
@pytest.mark.parametrize("dmin2,dmax2", [(1.0, np.inf), (0.0, np.inf), (25.0, 2500.0)])
def test_classes_make_the_same_traversal(kind, n, dims, dmin2, dmax2):
    pos4 = points(kind, n, dims)
    one, c1 = walk(pos4, dims, 1, dmin2, dmax2)
    # FP32 sums of at most n terms: each order is within n ulps of the terms' absolute sum, which
    # the largest velocity stands for here (terms of one sign along each axis from most points)
    scale = max(np.abs(one).max(), 1e-6)
    for group in (32, 16):
        v, c = walk(pos4, dims, group, dmin2, dmax2)
        assert c == c1
        np.testing.assert_allclose(v, one, rtol=0, atol=2e-5 * scale)
