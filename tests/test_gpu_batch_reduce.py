"""A batch's per-graph boxes and centre sums where a warp's 128 nodes, or a block's 1,024, hold one
graph, a few, or many, and graphs without nodes: every graph comes out as alone, bit for bit."""
import numpy as np
import pytest

from forcegpu.batch import Batch, GraphSpec
from forcegpu.graphs import benchmark_links

pytestmark = pytest.mark.gpu


def spec(n, dims, seed):
    rng = np.random.default_rng(seed)
    src, dst = benchmark_links(n, n // 2, seed=seed) if n > 1 else (None, None)
    return GraphSpec(xyz=rng.normal(seed % 7, 20, (n, dims)), source=src, target=dst)


@pytest.mark.parametrize("dims", [1, 2, 3])
@pytest.mark.parametrize("sizes", [[1, 2, 3, 0] * 60 + [127, 128, 129, 300], [31, 33, 0, 64, 1025, 5, 0, 0, 1023, 2],
                                   [4097, 128, 128, 128, 40, 40, 48], [2] * 700])
def test_every_graph_as_alone(sizes, dims):
    specs = [spec(n, dims, 100 + i) for i, n in enumerate(sizes)]
    mix = Batch()
    mix.set_graphs(specs, ndim=dims, seed=9)
    mix.run(3)
    pos, vel = mix.sync()
    mix.close()
    assert np.isfinite(pos).all()
    ends = np.cumsum(sizes)
    alone = Batch()
    for i in sorted({*range(0, len(sizes), 37), *range(len(sizes) - 4, len(sizes))}):
        if not sizes[i]:
            continue
        alone.set_graphs([specs[i]], ndim=dims, seed=9)
        alone.run(3)
        p, v = alone.sync()
        np.testing.assert_array_equal(p, pos[ends[i] - sizes[i]:ends[i]])
        np.testing.assert_array_equal(v, vel[ends[i] - sizes[i]:ends[i]])
    alone.close()
