"""A node object listed twice: it lands at its first place, and the other place sees that as an edit,
which goes up with the next tick (the nodes are landed one after the other in the reference,
src/gpu/engine.js:198-239)."""
import numpy as np

from test_host_mirror import mirror


def test_a_node_listed_twice_lands_once():
    a, b, c = ({"x": float(i), "y": 1.0, "vx": 0.0, "vy": 0.0} for i in range(3))
    m = mirror([a, b, a, c], 2)
    pos = np.arange(8, dtype=np.float32).reshape(4, 2) + np.float32(10.5)
    vel = -pos
    m.land(pos, vel)
    assert (a["x"], a["y"]) == (10.5, 11.5)
    assert (b["x"], c["x"]) == (12.5, 16.5)
    assert (a["vx"], a["vy"]) == (-14.5, -15.5)
    m.eng.calls.clear()
    m.sync_from_nodes()
    sent = [(args[0], args[1].tolist()) for name, args in m.eng.calls if name == "update_positions_packed"]
    assert sent == [(2, [[10.5, 11.5]])]
