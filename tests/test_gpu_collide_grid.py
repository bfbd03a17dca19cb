"""The collide grid's table of runs: every overlapping pair found once, whatever its cells, against
the Jacobi pushes in FP64; and words left from earlier ticks (their tag is the step's low 6 bits) not
taken for this tick's."""
import numpy as np
import pytest

from forcegpu._lib import Engine, desc_from_gpu

pytestmark = pytest.mark.gpu


def engine(pos4, vel4, dims, radii, iterations=1):
    n = len(pos4)
    e = Engine(0)
    e.set_nodes(pos4, dims, vel4=vel4)
    e.set_forces([desc_from_gpu({"type": "collide", "version": 1, "radii": radii, "strength": 0.7,
                                 "iterations": iterations}, 1, n)])
    e.set_seed(2)
    return e


def host(x, r, strength):
    """FP64 Jacobi pushes by pairs found along x; NaN for coincident nodes, whose push is d3's jiggle."""
    order = np.argsort(x[:, 0], kind="stable")
    push = np.zeros_like(x)
    reach = 2 * r.max()
    xs = x[order, 0]
    for a, i in enumerate(order):
        b = np.searchsorted(xs, xs[a] + reach, side="right")
        j = order[a + 1:b]
        d = x[i] - x[j]
        l = np.sqrt((d * d).sum(1))
        hit = l < r[i] + r[j]
        j, d, l = j[hit], d[hit], l[hit]
        with np.errstate(divide="ignore", invalid="ignore"):
            k = np.where(l > 0, (r[i] + r[j] - l) / l, np.nan) * strength
        t = r[i] ** 2 + r[j] ** 2
        push[i] += (d * (k * r[j] ** 2 / t)[:, None]).sum(0)
        np.add.at(push, j, -d * (k * r[i] ** 2 / t)[:, None])
    return push


@pytest.mark.parametrize("dims", [1, 2, 3])
@pytest.mark.parametrize("n,spread", [(8192, 6.0), (8193, 1.5), (20001, 3.0)])
def test_every_overlap_is_found_once(dims, n, spread):
    rng = np.random.default_rng(n + dims)
    pos4 = np.zeros((n, 4), np.float32)
    pos4[:, :dims] = rng.normal(-3, spread * n ** (1 / dims), (n, dims))
    radii = rng.uniform(0.5, 4, n).astype(np.float32)
    e = engine(pos4, None, dims, radii)
    e.enqueue(np.array([1.0]), 1.0)
    _, vel = e.sync()
    e.close()
    want = host(pos4[:, :dims].astype(np.float64), radii.astype(np.float64), 0.7)
    known = np.isfinite(want).all(1)
    assert known.mean() > 0.99 and np.abs(want[known]).max() > 0.1 and np.isfinite(vel).all()
    # a push is (r - l) / l of the distance: FP32 loses a few ulps of r (at most 8) against l, and a
    # node has at most some hundred of them
    np.testing.assert_allclose(vel[known, :dims], want[known], rtol=2e-4, atol=2e-4)


@pytest.mark.parametrize("dims,iterations", [(2, 1), (3, 2)])
def test_words_of_earlier_ticks_are_not_trusted(dims, iterations):
    n = 9001
    rng = np.random.default_rng(dims)
    pos4 = np.zeros((n, 4), np.float32)
    pos4[:, :dims] = rng.normal(0, 1.2 * n ** (1 / dims), (n, dims))
    vel4 = np.zeros((n, 4), np.float32)
    vel4[:, :dims] = rng.normal(0, 3, (n, dims))
    radii = rng.uniform(0.5, 2, n).astype(np.float32)
    e = engine(pos4, vel4, dims, radii, iterations)
    e.enqueue(np.full(140, 1.0), 0.99)
    pos, vel = e.sync()
    fresh = engine(pos, vel, dims, radii, iterations)
    for sim in (e, fresh):
        sim.enqueue(np.array([1.0]), 0.99)
    a, b = e.sync(), fresh.sync()
    e.close(), fresh.close()
    np.testing.assert_array_equal(a[0], b[0])
    np.testing.assert_array_equal(a[1], b[1])


@pytest.mark.parametrize("dims", [1, 2, 3])
@pytest.mark.parametrize("n", [2, 7, 8, 9, 33, 511, 512, 513, 1025, 8191])
def test_every_pair_of_a_small_layout(dims, n):
    """The pass over all pairs (below 8,192 nodes) at the edges of its blocks of 8 nodes and tiles of
    512, with the grid test's reference and tolerance."""
    rng = np.random.default_rng(n * 4 + dims)
    pos4 = np.zeros((n, 4), np.float32)
    pos4[:, :dims] = rng.normal(5, 2.0 * n ** (1 / dims), (n, dims))
    radii = rng.uniform(0.0, 4, n).astype(np.float32)
    radii[::11] = 0.0
    e = engine(pos4, None, dims, radii)
    e.enqueue(np.array([1.0]), 1.0)
    _, vel = e.sync()
    e.close()
    want = host(pos4[:, :dims].astype(np.float64), radii.astype(np.float64), 0.7)
    known = np.isfinite(want).all(1)
    assert np.isfinite(vel).all()
    np.testing.assert_allclose(vel[known, :dims], want[known], rtol=2e-4, atol=2e-4)
