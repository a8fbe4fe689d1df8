"""KNNSJ_VERBOSE=2 prints one line per search pass, also for joins searched
through the box tree: the lines' queries and failures add up to the join's
statistics."""
import re

import numpy as np
import pytest

import hybrid_k_nearest_neighbor_self_join_gb300 as kj
from hybrid_k_nearest_neighbor_self_join_gb300 import datasets

pytestmark = pytest.mark.gpu

LINE = re.compile(r"^knnsj: pass (\d+): (\d+) queries, (\d+) failed, .* ms, candidates so far (\d+)$", re.M)


@pytest.fixture(scope="module", autouse=True)
def built():
    import __graft_entry__
    __graft_entry__.build_library()


@pytest.mark.parametrize("tree", ["0", "1"])
@pytest.mark.parametrize("d,dtype,mode", [(3, np.float32, kj.RADIUS_PLAIN), (4, np.float32, kj.RADIUS_LEARNED),
                                          (5, np.float64, kj.RADIUS_PLAIN)])
def test_one_line_per_pass(monkeypatch, capfd, tree, d, dtype, mode):
    x = datasets.gmm(20_011, d, 9, 0.2, 600 + d, dtype=dtype)
    monkeypatch.setenv("KNNSJ_TREE", tree)
    ids, dists, quiet = kj.selfjoin(x, 24, radius_mode=mode, return_stats=True)
    capfd.readouterr()
    monkeypatch.setenv("KNNSJ_VERBOSE", "2")
    ids2, dists2, st = kj.selfjoin(x, 24, radius_mode=mode, return_stats=True)
    err = capfd.readouterr().err
    lines = [tuple(map(int, m)) for m in LINE.findall(err)]
    assert [m[0] for m in lines] == list(range(st["iterations"])), err
    assert lines[0][1] == len(x) and lines[-1][2] == 0
    assert all(a[2] == b[1] for a, b in zip(lines, lines[1:]))
    assert sum(m[1] for m in lines) == st["queries_run"]
    assert lines[-1][3] == st["candidates"]
    assert ("box tree" in err) == (tree == "1")
    # and nothing else changes
    assert np.array_equal(ids, ids2) and np.array_equal(dists, dists2)
    assert st["iterations"] == quiet["iterations"] and st["queries_run"] == quiet["queries_run"]
