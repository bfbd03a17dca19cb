"""The exact all-pairs sum with coordinates out of range: a source infinitely far (or so far that the
squared distance overflows) and a source without strength are left out, whatever their coordinates,
and a NaN with a strength reaches every node. One and two points per lane, with and without
distanceMax, against FP64 on the host."""
import numpy as np
import pytest

from forcegpu._lib import Engine, desc_from_gpu

pytestmark = pytest.mark.gpu


def run(pos4, dims, s, dmin2, dmax2):
    n = len(pos4)
    e = Engine(0)
    e.set_nodes(pos4, dims)
    e.set_forces([desc_from_gpu({"type": "manyBody", "version": 1, "strengths": s, "distanceMin2": dmin2,
                                 "distanceMax2": dmax2, "theta2": 0.0}, 1, n)])
    e.enqueue(np.array([0.5]), 1.0)
    _, vel = e.sync()
    e.close()
    return vel[:, :dims].astype(np.float64)


def host(x, s, alpha, dmin2, dmax2, rows):
    """FP64 sums and absolute sums; distances from dmax2 (or infinity) on are left out."""
    out, size = np.zeros((len(rows), x.shape[1])), np.zeros(len(rows))
    with np.errstate(invalid="ignore", over="ignore"):
        for k, i in enumerate(rows):
            d = x - x[i]
            l = (d * d).sum(1)
            ok = (np.arange(len(x)) != i) & (s != 0) & ~(l >= dmax2)
            d, l = d[ok], l[ok]
            w = s[ok] * alpha / np.where(l < dmin2, np.sqrt(dmin2 * l), l)
            out[k] = (d * w[:, None]).sum(0)
            size[k] = np.abs(d * w[:, None]).sum()
    return out, size


def layout(n, dims):
    rng = np.random.default_rng(n + dims)
    pos4 = np.zeros((n, 4), np.float32)
    for k in range(dims):  # distinct coordinates on every axis: no jiggle
        pos4[:, k] = rng.permutation(n) * 0.75 - 0.3 * n + rng.uniform(0, 0.25, n)
    return pos4, np.where(np.arange(n) % 5 == 0, 12.0, -30.0)


# a tile of its own, the tile of the checked rows and the last one
OUT = [(3, np.inf), (17, -np.inf), (36, 3e38), (-2, -3e38)]


@pytest.mark.parametrize("n", [40, 300, 10050])
@pytest.mark.parametrize("dims", [1, 2, 3])
@pytest.mark.parametrize("dmin2,dmax2", [(1.0, np.inf), (0.0, np.inf), (100.0, 250.0 ** 2)])
def test_sources_out_of_range_are_left_out(n, dims, dmin2, dmax2):
    pos4, s = layout(n, dims)
    for i, x in OUT:
        pos4[i, dims - 1] = x
    for i, x in ((9, np.nan), (21, np.inf), (-1, -np.inf)):  # without strength: as if not there
        pos4[i, 0], s[i] = x, 0.0
    s[5] = 0.0
    pos4[5, :dims] = pos4[6, :dims]
    if dims == 1:  # a subnormal squared distance, whose reciprocal overflows
        pos4[6, 0] = 0.0
        pos4[5, 0] = 1e-20
    v = run(pos4, dims, s, dmin2, dmax2)
    # node 5 itself meets node 6 at no distance (the jiggle's value) or, in 1D, too near for FP32
    inside = [i for i in range(n) if i != 5 and np.all(np.abs(pos4[i, :dims]) < 1e30)]
    rows = np.array(inside[:40] + inside[-40:])
    want, size = host(pos4[:, :dims].astype(np.float64), s, 0.5, dmin2, dmax2, rows)
    # FP32 terms and sums as in the sizes test: (8 + n / 32) half-ulps of the absolute sum; a source
    # within 2^-20 of distanceMax may fall on either side of it
    tol = (8 + n / 32) * 2.0 ** -24 * size[:, None] + 1e-6
    x = pos4[:, :dims].astype(np.float64)
    for k, i in enumerate(rows):
        with np.errstate(invalid="ignore", over="ignore"):
            l = ((x - x[i]) ** 2).sum(1)
        near = np.abs(l - dmax2) < 2.0 ** -20 * dmax2 if np.isfinite(dmax2) else np.zeros(n, bool)
        tol[k] += near.sum() * 30 * 0.5 / np.sqrt(dmax2) if near.any() else 0.0
    assert np.isfinite(v[inside]).all()
    assert np.all(np.abs(v[rows] - want) <= tol)
    # the nodes out of range meet no source at a finite distance
    for i, _ in OUT:
        np.testing.assert_array_equal(v[i], 0.0)


@pytest.mark.parametrize("n", [40, 10050])
@pytest.mark.parametrize("dmax2", [np.inf, 250.0 ** 2])
def test_two_nodes_at_one_infinity_meet_and_nobody_else(n, dmax2):
    pos4, s = layout(n, 3)
    pos4[3, 0] = pos4[30, 0] = np.inf
    v = run(pos4, 3, s, 1.0, dmax2)
    lost = ~np.isfinite(v).all(1)
    np.testing.assert_array_equal(np.flatnonzero(lost), [3, 30])  # inf - inf, as d3 has it


@pytest.mark.parametrize("n", [40, 10050])
def test_a_nan_with_a_strength_reaches_every_node(n):
    pos4, s = layout(n, 3)
    pos4[n // 2, 1] = np.nan
    v = run(pos4, 3, s, 1.0, np.inf)
    assert np.isnan(v).all()
