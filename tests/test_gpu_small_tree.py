"""The one-launch tree of a small layout at the edges of its runs of 256 points, its blocks' slices
(256, 512 and 768 points) and its clusters of 1 to 8 blocks, against the tree that digit passes and
separate launches build (asked for by the number of passes): the same sorted pairs, the same binary
tree and the same velocities bit for bit."""
import numpy as np
import pytest

from forcegpu._lib import TUNE_SORT_PASSES, Engine, desc_from_gpu

pytestmark = pytest.mark.gpu


def run(pos4, dims, charge, passes):
    n = len(pos4)
    e = Engine(0)
    e.set_nodes(pos4, dims)
    e.set_forces([desc_from_gpu({"type": "manyBody", "version": 1, "strengths": charge, "distanceMin2": 1.0,
                                 "distanceMax2": np.inf, "theta2": 0.81}, 1, n)])
    e.set_seed(3)
    e.set_tuning(TUNE_SORT_PASSES, passes)
    e.enqueue(np.array([0.7, 0.6]), 0.6)
    pos, vel = e.sync()
    tree = e.debug_tree(0)
    e.close()
    return [pos, vel, *tree]


@pytest.mark.parametrize("n,dims", [(2, 3), (3, 1), (255, 3), (256, 2), (257, 3), (511, 1), (513, 3), (1025, 2),
                                    (2047, 3), (2048, 3), (2049, 2), (3585, 3), (4096, 1), (4097, 3), (5377, 2),
                                    (6143, 3), (6144, 3)])
@pytest.mark.parametrize("kind", ["cloud", "places", "mixed"])
def test_one_launch_makes_the_tree_of_the_separate_passes(n, dims, kind):
    rng = np.random.default_rng(n)
    pos4 = np.zeros((n, 4), np.float32)
    pos4[:, :dims] = rng.integers(-5, 6, (n, dims)) if kind == "places" else rng.normal(0, 90, (n, dims))
    charge = np.where(np.arange(n) % 4 == 0, 12.0, -20.0) if kind == "mixed" else np.full(n, -30.0)
    for a, b in zip(run(pos4, dims, charge, 0), run(pos4, dims, charge, 4)):
        np.testing.assert_array_equal(a, b)
