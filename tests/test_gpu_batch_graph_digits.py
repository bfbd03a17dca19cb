"""A batch sorts its points by graph with one digit pass for up to 256 graphs and two for more: every
graph on both sides of that line comes out as alone, bit for bit."""
import numpy as np
import pytest

from forcegpu.batch import Batch, GraphSpec

pytestmark = pytest.mark.gpu


def run(sizes, first, last):
    b = Batch()
    b.set_graphs([GraphSpec(xyz=np.random.default_rng(i).normal(0, 30, (n, 3)))
                  for i, n in list(enumerate(sizes))[first:last]], ndim=3, seed=5)
    b.run(2)
    pos, vel = b.sync()
    b.close()
    return pos, vel


@pytest.mark.parametrize("graphs", [1, 2, 255, 256, 257, 513])
def test_every_graph_as_alone_on_both_sides_of_256_graphs(graphs):
    sizes = [2 + (37 * i) % 61 for i in range(graphs)]
    pos, vel = run(sizes, 0, graphs)
    ends = np.cumsum(sizes)
    for g in sorted({0, graphs // 2, max(graphs - 258, 0), max(graphs - 257, 0), max(graphs - 2, 0), graphs - 1}):
        p, v = run(sizes, g, g + 1)
        np.testing.assert_array_equal(p, pos[ends[g] - sizes[g]:ends[g]])
        np.testing.assert_array_equal(v, vel[ends[g] - sizes[g]:ends[g]])
