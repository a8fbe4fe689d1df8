"""Batched joins whose worker threads launch the same kernels with different
amounts of shared memory.

A kernel's dynamic shared memory limit is a property of the kernel, shared by
all host threads.  Sets of one dimension count and two values of k, and of
several dimension counts, make the tree's build and search kernels need
different amounts at the same time; with KNNSJ_TREE=0 the ring search does.
No set may be refused, and each set's rows are those of a single call.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

BODY = """
import numpy as np
import hybrid_k_nearest_neighbor_self_join_gb300 as kj
dt = np.dtype({dtype!r})
rng = np.random.default_rng(5)
ds = [2, 8, 3, 12, 8, 16]
xs = [rng.random((300 + 7 * i, ds[i % 6])).astype(dt) for i in range(96)]
ks = [{k_hi} if i // 6 % 2 else 4 for i in range(96)]
want = [kj.selfjoin(x, k) for x, k in zip(xs, ks)]
for _ in range(20):
    for (ids, dists), (wi, wd) in zip(kj.selfjoin_batched(xs, ks), want):
        assert np.array_equal(ids, wi)
        assert dists.tobytes() == wd.tobytes()
"""


@pytest.mark.parametrize("dtype,k_hi,tree", [("float32", 100, "1"), ("float64", 100, "1"), ("float32", 280, "0")])
def test_threads_launch_with_different_shared_memory(dtype, k_hi, tree):
    env = dict(os.environ, KNNSJ_TREE=tree, PYTHONPATH=ROOT)
    p = subprocess.run([sys.executable, "-c", BODY.format(dtype=dtype, k_hi=k_hi)], env=env, cwd=ROOT, timeout=300,
                       capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-2000:]
