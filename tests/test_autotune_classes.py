"""Batched joins try launch shapes only for classes whose search takes them.

The shapes belong to the grid's ring search.  Sets searched through the box
tree are not joined several times to pick one, and a class of ring-searched
sets is tuned also when sets of the same type, dimensions and k went through
the tree before it.  KNNSJ_VERBOSE=1 prints a line per join, trials included.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

BODY = """
import os, sys
import numpy as np
import hybrid_k_nearest_neighbor_self_join_gb300 as kj
from hybrid_k_nearest_neighbor_self_join_gb300 import datasets
os.environ["KNNSJ_VERBOSE"] = "1"
def batch(mode, d, dtype, n, tag, k=8):
    xs = [datasets.gmm(n + 100 * i, d, 6, 0.2, 40 + i, dtype=np.dtype(dtype)) for i in range(3)]
    print("== " + tag, file=sys.stderr, flush=True)
    kj.selfjoin_batched(xs, [k] * 3, radius_mode=mode)
"""


@pytest.fixture(scope="module", autouse=True)
def built():
    import __graft_entry__
    __graft_entry__.build_library()


def joins(body, tmp_path, **env):
    e = dict(os.environ, PYTHONPATH=ROOT, KNNSJ_TUNE_CACHE=str(tmp_path / "tune.txt"), **env)
    for name in ("KNNSJ_AUTOTUNE", "KNNSJ_VERBOSE", "KNNSJ_TREE"):
        e.pop(name, None)
    p = subprocess.run([sys.executable, "-c", BODY + body], env=e, cwd=ROOT, timeout=300, capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-2000:]
    out, tag = {}, None
    for line in p.stderr.splitlines():
        if line.startswith("== "):
            tag = line[3:]
            out[tag] = 0
        elif line.startswith("knnsj: n="):
            out[tag] += 1
    return out


def test_tree_classes_are_not_tried(tmp_path):
    got = joins("""
batch(kj.RADIUS_PLAIN, 4, "float32", 25_000, "plain")
batch(kj.RADIUS_LEARNED, 6, "float64", 25_000, "learned")
""", tmp_path)
    assert got == {"plain": 3, "learned": 3}


def test_ring_class_after_a_tree_class(tmp_path):
    # two-dimensional double sets: a uniform radius goes through the tree,
    # learned radii take the ring search below a million points
    body = """
batch(kj.RADIUS_PLAIN, 2, "float64", 25_000, "tree")
batch(kj.RADIUS_LEARNED, 2, "float64", 25_000, "ring")
batch(kj.RADIUS_LEARNED, 2, "float64", 25_000, "again")
"""
    got = joins(body, tmp_path)
    assert got["tree"] == 3 and got["again"] == 3
    assert got["ring"] > 3  # the warm-up and the shapes tried
    # a later process takes the ring class's shape from the file
    assert joins(body, tmp_path) == {"tree": 3, "ring": 3, "again": 3}


def test_rows_too_long_for_the_tree_are_tried(tmp_path):
    # k+1 above 224: the ring search, in a class of its own
    got = joins('batch(kj.RADIUS_PLAIN, 3, "float32", 25_000, "long", k=240)\n', tmp_path)
    assert got["long"] > 3
