"""A tree whose root claims child slots that are not there (tests/c/malformed_tree.cu, linked to the
engine's objects): the walk marks it, drops the entry and ends, instead of walking on from the root
until its guard on the rounds."""
import glob
import itertools
import os
import subprocess
import sys

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu

TREE = 4  # FL_ERR_TREE, without FL_ERR_STACK


def test_an_entry_past_the_slots_is_dropped(tmp_path):
    sys.path.insert(0, PKG)
    import build
    build.build()
    exe = str(tmp_path / "malformed_tree")
    objects = sorted(glob.glob(os.path.join(PKG, "_build", "*.o")))
    subprocess.check_call([build.nvcc(), os.path.join(ROOT, "tests", "c", "malformed_tree.cu"), "-o", exe,
                           "-std=c++17", "--expt-relaxed-constexpr"] + build.ARCH + objects)
    cases = list(itertools.product([4, 100, 3000], [1, 16, 32], [1, 2, 3], [(1, 1 << 20), (0xffffffff, 1), (0x7fffffff, 40), (1, 0)]))
    args = [str(a) for n, group, dims, (first, count) in cases for a in (n, group, dims, first, count)]
    r = subprocess.run([exe] + args, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
    lines = r.stdout.split("\n")[:-1]
    assert len(lines) == len(cases)
    for (n, group, *_), line in zip(cases, lines):
        err, tests = map(int, line.split())
        assert err == TREE
        # two rounds a traversal (the root, the entry in its place), a child each, per point
        points = n if group == 1 else group * -(-n // group)
        assert tests <= 2 * points
