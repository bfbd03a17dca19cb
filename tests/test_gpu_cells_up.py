"""The recursion of cells with charges of both signs gives every warp 128 consecutive binary nodes
and counts the cells within them apart from the cells above. A graph's place in a batch moves those
boundaries through its tree, and none of its results: it comes out as alone, bit for bit. (Among the
2,500 points on 7 places of a line one pair draws a jiggle of 0, and d3's x / 0 makes that graph NaN.)"""
import numpy as np
import pytest

from forcegpu.batch import Batch, GraphSpec

pytestmark = pytest.mark.gpu


def spec(n, dims, kind):
    rng = np.random.default_rng(n)
    # "grid": many points on one place, a deepest cell with more children than a warp has nodes
    x = rng.integers(-3, 4, (n, dims)) if kind == "grid" else rng.normal(0, 40, (n, dims))
    return GraphSpec(xyz=np.float32(x), charge=np.where(np.arange(n) % 4 == 0, 12.0, -20.0))


@pytest.mark.parametrize("kind,dims", [("cloud", 3), ("cloud", 2), ("grid", 3), ("grid", 1)])
@pytest.mark.parametrize("n", [2, 127, 129, 513, 2500])
def test_a_graph_comes_out_the_same_wherever_its_nodes_lie(n, dims, kind):
    me, out = spec(n, dims, kind), []
    for before in ([], [1], [126], [127], [128], [129, 2], [511], [1000, 31]):
        b = Batch()
        b.set_graphs([spec(k, dims, "cloud") for k in before] + [me, spec(33, dims, "cloud")], ndim=dims, seed=3)
        b.run(2)
        out.append(b.read(len(before)))
        b.close()
    for pos, vel in out:
        np.testing.assert_array_equal(pos, out[0][0])
        np.testing.assert_array_equal(vel, out[0][1])
