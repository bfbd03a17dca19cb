"""The exact all-pairs sum with a distanceMax that cuts through the layout, so that every node has many
sources on either side of it: against FP64, with an allowance only for the rows that have a source
within rounding of the cutoff."""
import numpy as np
import pytest

from test_gpu_allpairs_sizes import host, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 129, 1025, 4099, 10000, 10001, 12289])
@pytest.mark.parametrize("dims", [1, 2, 3])
def test_sources_on_both_sides_of_the_cutoff(n, dims):
    rng = np.random.default_rng(n * 4 + dims)
    pos4 = np.zeros((n, 4), np.float32)
    for k in range(dims):  # distinct coordinates on every axis within +-100: no jiggle
        pos4[:, k] = (rng.permutation(n) + rng.uniform(0, 0.3, n)) * (200.0 / n) - 100.0
    s = np.where(np.arange(n) % 5 == 0, 12.0, -30.0)
    s[n // 2] = 0.0
    dmin2, dmax2 = 9.0, 100.0 ** 2
    v = run(pos4, dims, s, dmin2, dmax2)
    rows = np.unique(np.concatenate([np.arange(min(n, 40)), np.arange(max(0, n - 40), n), rng.integers(0, n, 40)]))
    x = pos4[:, :dims].astype(np.float64)
    want, size = host(x, s, 0.5, dmin2, dmax2, rows)
    l = ((x[None] - x[rows][:, None]) ** 2).sum(2)
    inside = (l < dmax2).mean(1)
    assert np.mean((inside > 0.1) & (inside < 0.9)) > 0.6  # the cutoff does cut
    # FP32 terms and sums as in the sizes test; l carries at most 4 roundings, 2^-22 of it
    tol = (8 + n / 32) * 2.0 ** -24 * size + 1e-6
    tol += (np.abs(l - dmax2) < 2.0 ** -21 * dmax2).sum(1) * 30 * 0.5 / 100.0
    assert np.all(np.abs(v[rows] - want) <= tol[:, None])
