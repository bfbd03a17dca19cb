"""The host mirror's reading and landing of nodes, and the force arrays it does not send again,
against a fake engine (no GPU): every kind of value a node may hold, as the reference's engine takes
it (src/gpu/engine.js:61-63, :115-239)."""
import math
from collections import defaultdict

import numpy as np
import pytest

from forcegpu import forceCenter, forceLink, forceManyBody
from forcegpu._lib import desc_from_gpu
from forcegpu.simulation import _NodeMirror, _num


class FakeEngine:
    def __init__(self):
        self.calls, self.refuse = [], False

    def __getattr__(self, name):
        return lambda *a, **k: self.calls.append((name, a))

    def set_forces(self, descs):
        if self.refuse:
            raise RuntimeError("refused")
        self.calls.append(("set_forces", [(d.node_a, d.source, d.m, d.version) for d, _ in descs]))


def mirror(nodes, dims):
    m = _NodeMirror.__new__(_NodeMirror)
    m.eng = FakeEngine()
    m.stale, m.plan, m.sent = False, [], {}
    m.set_nodes(nodes, dims)
    return m


ODD = [1, 2.5, None, math.nan, "3.5", "x", True, np.float64(4.5), np.float32(0.25), -0.0, math.inf, 10 ** 30]


@pytest.mark.parametrize("dims", [1, 2, 3])
def test_reading_takes_every_kind_of_value_as_before(dims):
    nodes = [{"x": v, "y": w} for v in ODD for w in ODD] + [{}, defaultdict(float)]
    nodes[3]["fx"], nodes[5]["fy"], nodes[7]["fx"] = 2, np.float32(1.5), None
    m = mirror(nodes, dims)
    pos, fix, mask = m._read(0, len(nodes))
    axes = "xyz"[:dims]
    for i, node in enumerate(nodes):
        for k in range(3):
            want = _num(node.get("xyz"[k])) if k < dims else 0.0
            assert pos[i, k] == want
            pin = node.get("f" + "xyz"[k]) if k < dims else None
            assert bool(mask[i] >> k & 1) == (pin is not None)
            assert fix[i, k] == (0.0 if pin is None else float(pin))
    assert nodes[-1] == {} and axes  # reading adds nothing to a node


def test_landing_keeps_what_the_user_changed():
    nodes = [{"x": float(i), "y": 0.5, "vx": 0.0, "vy": 0.0} for i in range(50)]
    m = mirror(nodes, 2)
    nodes[7]["x"] = 100.0
    nodes[9]["y"] = None
    pos = np.arange(100, dtype=np.float32).reshape(50, 2) + np.float32(0.1)
    vel = -pos
    m.land(pos, vel)
    for i, node in enumerate(nodes):
        assert (node["vx"], node["vy"]) == (float(vel[i, 0]), float(vel[i, 1]))
        if i == 7:
            assert node["x"] == 100.0 and node["y"] == 0.5
        elif i == 9:
            assert node["x"] == 9.0 and node["y"] is None
        else:
            assert (node["x"], node["y"]) == (float(pos[i, 0]), float(pos[i, 1]))
            assert type(node["x"]) is float
    m.sync_from_nodes()  # the two edits go up, nothing else
    sent = [a[0] for name, a in m.eng.calls if name == "update_positions_packed"]
    assert sent == [7, 9]
    del nodes[40:]  # fewer nodes than the simulation was given: those that are left land
    m.land(pos, vel)
    assert nodes[39]["vx"] == float(vel[39, 0])
    nodes += [{"x": 0.0, "y": 0.0}] * 11
    with pytest.raises(IndexError):
        m.land(pos, vel)


def test_arrays_are_sent_once_per_version():
    nodes = [{"x": float(i), "index": i} for i in range(5)]
    m = mirror(nodes, 3)
    charge, links, center = forceManyBody(), forceLink([{"source": 0, "target": 1}]), forceCenter()
    for f in (charge, links, center):
        f.initialize(nodes, None, 3)

    def arrays():
        m.set_forces([charge, links, center])
        return [(bool(a), bool(s), mm) for a, s, mm, _ in m.eng.calls[-1][1]]

    assert arrays() == [(True, False, 0), (False, True, 1), (False, False, 0)]
    assert arrays() == [(False, False, 0), (False, False, 1), (False, False, 0)]
    charge.strength(-5)
    assert arrays()[0][0] is True
    assert arrays()[0][0] is False
    m.eng.refuse = True  # a refused call leaves the engine without passes: everything again
    with pytest.raises(RuntimeError):
        m.set_forces([charge, links, center])
    m.eng.refuse = False
    assert arrays() == [(True, False, 0), (False, True, 1), (False, False, 0)]
    m.set_nodes(nodes, 3)  # a new node set forgets the forces
    assert arrays() == [(True, False, 0), (False, True, 1), (False, False, 0)]
    m.set_forces([charge, charge])  # one object twice is two passes
    assert [bool(a) for a, *_ in m.eng.calls[-1][1]] == [True, True]


def test_scalars_are_the_same_without_arrays():
    nodes = [{"index": i} for i in range(4)]
    links = forceLink([{"source": 0, "target": 1}, {"source": 2, "target": 1}]).iterations(3)
    links.initialize(nodes, None, 3)
    for g in (links.gpu(), {"type": "link", "version": 4, "source": [0], "target": [1], "iterations": 2,
                            "strengths": [1.0], "distances": [1.0], "bias": [0.5]}):
        a, b = desc_from_gpu(g, 9, 4)[0], desc_from_gpu(g, 9, 4, arrays=False)[0]
        assert (a.m, a.iterations, a.version, a.key, a.type) == (b.m, b.iterations, b.version, b.key, b.type)
        assert not b.source and not b.link_bias
