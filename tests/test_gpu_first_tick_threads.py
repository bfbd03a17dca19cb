"""The first ticks of a process, of several simulations at once from threads of their own: a layout
whose kernels take more shared memory than a block may have by default (the tree in one launch, and a
sort by digits) runs in each, and gives what one alone gives. Each try is a fresh process: the
kernels' limits are raised once."""
import subprocess
import sys

import pytest

from conftest import PKG

FIRST = """
import sys, threading
sys.path.insert(0, %r)
import numpy as np
from forcegpu._lib import Engine, desc_from_gpu
n, threads = int(sys.argv[1]), 16
pos = np.zeros((n, 4), np.float32)
pos[:, :3] = np.random.default_rng(1).normal(0, 50, (n, 3))
charge = {"type": "manyBody", "version": 1, "strengths": np.full(n, -30.0), "distanceMin2": 1.0,
          "distanceMax2": np.inf, "theta2": 0.81}
engines = [Engine(0) for _ in range(threads)]
for e in engines:
    e.set_nodes(pos, 3)
    e.set_forces([desc_from_gpu(charge, 1, n)])
    e.set_seed(1)
gate, out = threading.Barrier(threads), [None] * threads

def tick(i):
    gate.wait()
    try:
        engines[i].enqueue([0.5], 0.6)
        out[i] = engines[i].sync()[0]
    except Exception as x:
        out[i] = x

ts = [threading.Thread(target=tick, args=(i,)) for i in range(threads)]
[t.start() for t in ts]
[t.join() for t in ts]
for r in out:
    if isinstance(r, Exception):
        sys.exit(str(r))
    if not np.array_equal(r, out[0]) or not np.isfinite(r).all():
        sys.exit("the threads' results differ")
"""


@pytest.mark.gpu
@pytest.mark.parametrize("n", [6000, 200_000])
def test_threads_may_make_the_first_ticks_together(n):
    for _ in range(4):
        r = subprocess.run([sys.executable, "-c", FIRST % PKG, str(n)], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stderr[-2000:]
