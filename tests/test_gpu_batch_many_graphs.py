"""The per-graph values of a batch come from a warp per graph up to a few hundred graphs and from a
thread per graph beyond: a graph of a large batch comes out as in a small one, bit for bit, whatever
the extent of its cube (none, less than 1, powers of two, the largest, a coordinate that is no number)."""
import numpy as np
import pytest

from forcegpu.batch import Batch, GraphSpec

pytestmark = pytest.mark.gpu

EXTENTS = [0.0, 0.3, 1.0, 2.0, 64.0, 1000.0, 3e7, 1e20, 1e38, np.inf, np.nan]


def spec(i, dims):
    rng = np.random.default_rng(i)
    x = rng.uniform(-0.5, 0.5, (1 + i % 7, dims))
    x[0] = 0.0
    e = EXTENTS[i % len(EXTENTS)]
    if np.isfinite(e):
        x *= e
    else:
        x[-1, i % dims] = e
    return GraphSpec(xyz=np.float32(x), charge=-30.0, center=(1.0, 2.0, 3.0))


def run(specs, dims):
    b = Batch()
    b.set_graphs(specs, ndim=dims, seed=3)
    b.run(2)
    out = [b.read(i) for i in range(len(specs))]
    b.close()
    return out


@pytest.mark.parametrize("dims", [1, 2, 3])
@pytest.mark.parametrize("graphs", [601, 700, 2050])
def test_a_graph_of_many_comes_out_as_one_of_few(graphs, dims):
    specs = [spec(i, dims) for i in range(graphs)]
    few = [r for k in range(0, graphs, 100) for r in run(specs[k:k + 100], dims)]
    for (p, v), (q, w) in zip(run(specs, dims), few):
        np.testing.assert_array_equal(p, q)
        np.testing.assert_array_equal(v, w)
