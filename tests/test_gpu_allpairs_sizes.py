"""The exact all-pairs sum at the edges of its tiles (32 sources, 4 at a time), of its two forms
(one or two points per lane, from 10,001 points) and of its clusters, against FP64 on the host; with
the cases that leave its common path: coincident points, a shared coordinate, distanceMin and
distanceMax."""
import numpy as np
import pytest

from forcegpu._lib import Engine, desc_from_gpu

pytestmark = pytest.mark.gpu


def host(x, s, alpha, dmin2, dmax2, rows):
    """FP64 sums for the given rows, and each row's absolute sum; no zero components."""
    out, size = np.zeros((len(rows), x.shape[1])), np.zeros(len(rows))
    for k, i in enumerate(rows):
        d = x - x[i]
        l = (d * d).sum(1)
        ok = (np.arange(len(x)) != i) & (l < dmax2)
        d, l = d[ok], l[ok]
        w = s[ok] * alpha / np.where(l < dmin2, np.sqrt(dmin2 * l), l)
        out[k] = (d * w[:, None]).sum(0)
        size[k] = np.abs(d * w[:, None]).sum()
    return out, size


def run(pos4, dims, s, dmin2, dmax2):
    n = len(pos4)
    e = Engine(0)
    e.set_nodes(pos4, dims)
    e.set_forces([desc_from_gpu({"type": "manyBody", "version": 1, "strengths": s, "distanceMin2": dmin2,
                                 "distanceMax2": dmax2, "theta2": 0.0}, 1, n)])
    e.set_seed(5)
    e.enqueue(np.array([0.5]), 1.0)
    _, vel = e.sync()
    e.close()
    return vel[:, :dims].astype(np.float64)


@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 63, 129, 1025, 4099, 10000, 10001, 12289])
@pytest.mark.parametrize("dims", [1, 2, 3])
@pytest.mark.parametrize("dmin2,dmax2", [(1.0, np.inf), (400.0, 40000.0)])
def test_against_fp64(n, dims, dmin2, dmax2):
    rng = np.random.default_rng(n * 4 + dims)
    pos4 = np.zeros((n, 4), np.float32)
    # distinct coordinates on every axis: no jiggle
    for k in range(dims):
        pos4[:, k] = rng.permutation(n) * 0.75 - 0.3 * n + rng.uniform(0, 0.25, n)
    s = np.where(np.arange(n) % 5 == 0, 12.0, -30.0)
    s[n // 2] = 0.0
    v = run(pos4, dims, s, dmin2, dmax2)
    rows = np.unique(np.concatenate([np.arange(min(n, 40)), np.arange(max(0, n - 40), n), rng.integers(0, n, 40)]))
    x = pos4[:, :dims].astype(np.float64)
    want, size = host(x, s, 0.5, dmin2, dmax2, rows)
    # FP32 terms (4 roundings and a reciprocal within 1 ulp: 8 ulps with margin) and sums of n / 32
    # terms per partial at most: within (8 + n / 32) half-ulps of the absolute sum, and a source
    # within rounding of distanceMax may fall on either side of it: one term of 30 * alpha / d
    edge = 0.0 if dmax2 == np.inf else 30 * 0.5 / np.sqrt(dmax2)
    tol = (8 + n / 32) * 2.0 ** -24 * size[:, None] + 2 * edge + 1e-6
    assert np.all(np.abs(v[rows] - want) <= tol)


@pytest.mark.parametrize("n", [40, 10050])
def test_coincident_points_and_shared_coordinates(n):
    rng = np.random.default_rng(n)
    pos4 = np.zeros((n, 4), np.float32)
    pos4[:, :3] = rng.normal(0, 50, (n, 3))
    pos4[10:14] = pos4[9]        # coincident: d3's jiggle, antisymmetric
    pos4[20:30, 1] = pos4[19, 1]  # a zero component only
    v = run(pos4, 3, np.full(n, -30.0), 1.0, np.inf)
    assert np.isfinite(v).all()
    assert len(np.unique(v[9:14], axis=0)) == 5  # the jiggle parts them
    again = run(pos4, 3, np.full(n, -30.0), 1.0, np.inf)
    np.testing.assert_array_equal(v, again)
    # action equals reaction: the sum over all points vanishes up to rounding
    assert np.all(np.abs(v.sum(0)) <= 1e-4 * np.abs(v).sum())
