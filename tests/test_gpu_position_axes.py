"""Position forces that follow one another: different axes in one launch, an axis again in its own, an
axis that the layout does not have left out. The sums are the forces' own, one after the other."""
import numpy as np
import pytest

from forcegpu._lib import Engine, desc_from_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,axes", [(3, [0, 1, 2]), (3, [2, 0, 0, 1]), (2, [0, 2, 1]), (2, [1, 1, 0]), (1, [2, 0, 1]),
                                       (2, [2])])
@pytest.mark.parametrize("n", [1, 257])
def test_forces_of_several_axes(n, dims, axes):
    rng = np.random.default_rng(n)
    pos4 = np.zeros((n, 4), np.float32)
    pos4[:, :dims] = rng.normal(0, 50, (n, dims))
    target, strength = rng.normal(0, 30, (len(axes), n)), rng.uniform(0.05, 0.4, (len(axes), n))
    e = Engine(0)
    e.set_nodes(pos4, dims)
    e.set_forces([desc_from_gpu({"type": "position", "version": 1, "axis": a, "targets": t, "strengths": s}, 1, n)
                  for a, t, s in zip(axes, target, strength)])
    e.enqueue(np.array([0.7]), 1.0)  # no decay: the velocity is the sum of the forces
    _, vel = e.sync()
    e.close()
    want = np.zeros((n, 4))
    for a, t, s in zip(axes, target, strength):
        if a < dims:
            want[:, a] += (t - pos4[:, a]) * s * 0.7
    # each term: three roundings and those of its target and strength, 5 ulps of |target| + |p| at most
    atol = 5 * 2.0 ** -23 * len(axes) * (np.abs(target).max() + np.abs(pos4).max())
    np.testing.assert_allclose(vel, want, rtol=0, atol=atol)
