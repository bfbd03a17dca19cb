"""Coincident nodes whose jiggle draws the middle of its range: they part, by equal and opposite
amounts, in every force that draws one; and a deepest cell of charges of both signs with more points
than the recursion's warps have nodes, among which such a draw happens."""
import numpy as np
import pytest

from forcegpu._lib import Engine, desc_from_gpu
from forcegpu.batch import Batch, GraphSpec

SEEDS = [10451126, 54968099, 101339792, 115772319]  # nodes 0 and 1, axis 0, step 0


def mix32(x):
    x ^= x >> 16
    x = x * 0x7feb352d & 0xffffffff
    x ^= x >> 15
    x = x * 0x846ca68b & 0xffffffff
    return x ^ x >> 16


@pytest.mark.parametrize("seed", SEEDS)
def test_the_seeds_draw_the_middle(seed):
    h = mix32(0 ^ mix32(1 ^ mix32(seed ^ mix32(0))))
    assert np.float32(h) == np.float32(2 ** 31) and -64 <= h - 2 ** 31 <= 128


def force(kind):
    if kind == "collide":
        return {"type": "collide", "version": 1, "radii": np.full(2, 3.0), "strength": 1.0, "iterations": 1}
    return {"type": "manyBody", "version": 1, "strengths": np.full(2, -30.0), "distanceMin2": 1.0,
            "distanceMax2": np.inf, "theta2": 0.0 if kind == "exact" else 0.81}


@pytest.mark.gpu
@pytest.mark.parametrize("seed", SEEDS)
@pytest.mark.parametrize("kind", ["charge", "exact", "collide"])
def test_two_nodes_on_one_place_part(kind, seed):
    e = Engine(0)
    e.set_nodes(np.zeros((2, 4), np.float32), 1)
    e.set_forces([desc_from_gpu(force(kind), 1, 2)])
    e.set_seed(seed)
    e.enqueue(np.array([0.5]), 1.0)
    _, vel = e.sync()
    e.close()
    assert np.isfinite(vel).all() and vel[0, 0] != 0.0
    assert vel[0, 0] == -vel[1, 0]


def crowd(dims, places, each, seed):
    rng = np.random.default_rng(seed)
    x = np.repeat(rng.permutation(3 ** dims * 9)[:places, None] // 3 ** np.arange(dims) % 9, each, 0)
    return np.float32(x[rng.permutation(len(x))])


@pytest.mark.gpu
@pytest.mark.parametrize("dims,places,each", [(1, 7, 300), (2, 5, 129), (3, 8, 300), (3, 2, 1000)])
def test_crowded_places_of_both_signs_stay_finite(dims, places, each):
    x = crowd(dims, places, each, dims + each)
    me, out = GraphSpec(xyz=x, charge=np.where(np.arange(len(x)) % 4 == 0, 12.0, -20.0)), []
    for before in (0, 1, 127, 500):
        b = Batch()
        b.set_graphs([GraphSpec(xyz=np.random.default_rng(1).normal(0, 9, (before, dims)).astype(np.float32),
                                charge=-30.0)] * (before > 0) + [me], ndim=dims, seed=3)
        b.run(2)
        out.append(b.read(int(before > 0)))
        b.close()
    for pos, vel in out:
        assert np.isfinite(pos).all() and np.isfinite(vel).all()
        np.testing.assert_array_equal(pos, out[0][0])
        np.testing.assert_array_equal(vel, out[0][1])


@pytest.mark.gpu
def test_a_crowd_with_a_draw_of_the_middle_stays_finite():
    x = np.random.default_rng(2500).integers(-3, 4, (2500, 1))  # one pair of it draws the middle
    b = Batch()
    b.set_graphs([GraphSpec(xyz=np.float32(x), charge=np.where(np.arange(2500) % 4 == 0, 12.0, -20.0))], ndim=1, seed=3)
    b.run(2)
    pos, vel = b.read(0)
    b.close()
    assert np.isfinite(pos).all() and np.isfinite(vel).all()
