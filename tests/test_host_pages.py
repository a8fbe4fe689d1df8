"""Result tables into ordinary host arrays, whether or not their pages are in
memory yet.

Fresh arrays are filled by several threads, which take the page faults side by
side; arrays in use (up to 128 MB) by the runtime's copy, which is faster there.
The choice is by the pages in memory (csrc/host_pages.h).
"""
import mmap
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_absent_bytes(tmp_path):
    exe = tmp_path / "host_pages_check"
    subprocess.check_call(["g++", "-O1", "-std=c++17",
                           "-I", os.path.join(ROOT, "hybrid_k_nearest_neighbor_self_join_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "host_pages_check.cpp"), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and "bad=0" in out.stdout, out.stdout


def fresh(shape, dtype):
    return np.frombuffer(mmap.mmap(-1, int(np.prod(shape)) * np.dtype(dtype).itemsize), dtype).reshape(shape)


@pytest.mark.gpu
@pytest.mark.parametrize("touched", [0.0, 0.3, 0.9, 1.0])
@pytest.mark.parametrize("n,k,dtype", [(40_001, 16, np.float32), (300_007, 8, np.float64)])
def test_rows(touched, n, k, dtype):
    import __graft_entry__
    import hybrid_k_nearest_neighbor_self_join_gb300 as kj
    from hybrid_k_nearest_neighbor_self_join_gb300 import datasets
    __graft_entry__.build_library()
    x = datasets.gmm(n, 2, 7, 0.2, n, dtype=dtype)
    want = kj.selfjoin(x, k)
    ids, dists = fresh((n, k + 1), np.int32), fresh((n, k + 1), dtype)
    for a in (ids, dists):
        a.reshape(-1)[:int(a.size * touched)] = -1
    kj.selfjoin(x, k, out_ids=ids, out_dists=dists)
    assert np.array_equal(ids, want[0]) and dists.tobytes() == want[1].tobytes()


@pytest.mark.gpu
def test_warm_arrays_are_not_staged():
    # 128 MB of rows into warm arrays: 0.8 ms by the runtime's copy at the link's
    # rate, 2.2 staged; the best of several calls against other load on the host
    import __graft_entry__
    import hybrid_k_nearest_neighbor_self_join_gb300 as kj
    from hybrid_k_nearest_neighbor_self_join_gb300 import datasets
    __graft_entry__.build_library()
    n, k = 500_000, 31
    x = datasets.uniform(n, 2, 5)
    ids, dists = np.zeros((n, k + 1), np.int32), np.zeros((n, k + 1), np.float32)
    best = min(kj.selfjoin(x, k, radius_mode=kj.RADIUS_LEARNED, out_ids=ids, out_dists=dists,
                           return_stats=True)[2]["ms_transfer"] for _ in range(12))
    assert best < 1.4, best
