"""The memory that fl_fits counts for a layout is no less than what a layout with a charge and a
collide force takes."""
import ctypes

import numpy as np
import pytest

from forcegpu._lib import Engine, desc_from_gpu, load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1000, 70_000, 2_100_000])
def test_a_layout_takes_no_more_than_is_counted(n):
    torch = pytest.importorskip("torch")
    layout_bytes = getattr(load(), "_Z15fl_layout_bytesl")  # the engine's own, not part of the C ABI
    layout_bytes.restype, layout_bytes.argtypes = ctypes.c_int64, [ctypes.c_int64]
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = np.random.default_rng(1).normal(0, 8 * n ** (1 / 3), (n, 3))
    charge = {"type": "manyBody", "version": 1, "strengths": np.full(n, -30.0), "distanceMin2": 1.0,
              "distanceMax2": np.inf, "theta2": 0.81}
    collide = {"type": "collide", "version": 1, "radii": np.full(n, 2.0), "strength": 0.7, "iterations": 1}
    e = Engine(0)
    e.idle()
    before = torch.cuda.mem_get_info()[0]
    e.set_nodes(pos, 3)
    e.set_forces([desc_from_gpu(charge, 1, n), desc_from_gpu(collide, 2, n)])
    e.idle()
    used = before - torch.cuda.mem_get_info()[0]
    e.close()
    assert used <= layout_bytes(n) + 16 * (2 << 20)  # some 16 buffers, in whole pages of 2 MB
