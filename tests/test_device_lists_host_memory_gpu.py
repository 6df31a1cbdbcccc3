"""Leaf lists built on the device reach the host without the pool they lie in (B200)."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import sys
sys.path[:0] = [{root!r}, {tests!r}]
import conftest
import gx

def peak():
    with open("/proc/self/status") as f:
        return next(int(line.split()[1]) for line in f if line.startswith("VmHWM")) * 1024

args = dict(softening=0.02, theta=0.9, leaf_capacity=8, on_device=True)
small = gx.ics.two_disk_encounter(500, 500, 3, 0.02)
gx.build_leaf_lists(small.x, small.y, small.z, small.m, **args)
p = gx.ics.two_disk_encounter(1 << 17, 1 << 17, 3, 0.02)
before = peak()
lists = gx.build_leaf_lists(p.x, p.y, p.z, p.m, **args)
assert lists.built_on_device
print(peak() - before, sum(a.nbytes for a in (lists.leaf_offsets, lists.leaf_particles, lists.near_offsets,
                                               lists.near_leaves)), lists.n_leaves)
"""


def test_host_memory_follows_the_lists():
    """The pool holds 1 KiB of near list per leaf with bodies, at theta 0.9 most of it unused; the
    host needs the lists twice (the tree's and the caller's) and a few words per leaf."""
    tests = Path(__file__).resolve().parent
    out = subprocess.run([sys.executable, "-c", CHILD.format(root=str(tests.parent), tests=str(tests))], check=True,
                         capture_output=True, text=True, timeout=300).stdout
    grown, lists, leaves = map(int, out.split())
    assert lists < 1024 * leaves / 2
    assert grown <= 2 * lists + 64 * leaves + (16 << 20)
