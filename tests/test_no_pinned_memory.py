"""Joins on a host that grants no page-locked memory.

The library keeps a few blocks of it for small reads, the dimension sample and
result tables on their way into ordinary arrays; none of them is needed for an
answer.  KNNSJ_TEST_PINNED_KB makes the library refuse itself larger blocks,
from the first call of a process on.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

BODY = """
import sys
import numpy as np, torch
import hybrid_k_nearest_neighbor_self_join_gb300 as kj
from hybrid_k_nearest_neighbor_self_join_gb300 import datasets
out = {}
for i, (n, d, k, dt, mode) in enumerate([(30_000, 2, 8, np.float32, 1), (20_000, 4, 16, np.float64, 0),
                                         (300_000, 2, 8, np.float32, 0), (900, 3, 5, np.float32, 0)]):
    x = datasets.gmm(n, d, 7, 0.2, 50 + i, dtype=dt)
    out[f"h{i}"], out[f"hd{i}"] = kj.selfjoin(x, k, radius_mode=mode)
    t = torch.from_numpy(x).cuda()
    ids = torch.empty(n, k + 1, dtype=torch.int32, device="cuda")
    dists = torch.empty(n, k + 1, dtype=t.dtype, device="cuda")
    torch.cuda.synchronize()
    kj.selfjoin_device(t.data_ptr(), dt, n, d, k, ids.data_ptr(), dists.data_ptr(), radius_mode=mode)
    out[f"d{i}"], out[f"dd{i}"] = ids.cpu().numpy(), dists.cpu().numpy()
xs = [datasets.gmm(4_000 + 900 * i, 3, 5, 0.2, 80 + i, dtype=np.float32) for i in range(5)]
for i, (a, b) in enumerate(kj.selfjoin_batched(xs, [6] * 5)):
    out[f"b{i}"], out[f"bd{i}"] = a, b
np.savez(sys.argv[1], **out)
"""


@pytest.fixture(scope="module", autouse=True)
def built():
    import __graft_entry__
    __graft_entry__.build_library()


def rows(path, **env):
    np = pytest.importorskip("numpy")
    p = subprocess.run([sys.executable, "-c", BODY, str(path)], env=dict(os.environ, PYTHONPATH=ROOT, **env), cwd=ROOT,
                       timeout=300, capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-2000:]
    return np.load(path)


@pytest.mark.parametrize("kb", ["0", "20"])
def test_same_rows(tmp_path, kb):
    want = rows(tmp_path / "want.npz")
    got = rows(tmp_path / "got.npz", KNNSJ_TEST_PINNED_KB=kb)
    assert sorted(want) == sorted(got)
    for name in want:
        assert want[name].tobytes() == got[name].tobytes(), name


def test_largest_block():
    # the blocks a workspace keeps are at most 16 MB, whatever the size of the
    # data: here the dimension sample alone has 32 MB
    body = """
import numpy as np, torch
import hybrid_k_nearest_neighbor_self_join_gb300 as kj
n = 200_000_000
g = torch.Generator(device="cuda"); g.manual_seed(1)
x = torch.rand(n, 2, generator=g, device="cuda", dtype=torch.float64)
x[:, 1] *= 1.5
ids = torch.empty(n, 2, dtype=torch.int32, device="cuda")
dists = torch.empty(n, 2, dtype=x.dtype, device="cuda")
torch.cuda.synchronize()
st = kj.selfjoin_device(x.data_ptr(), np.float64, n, 2, 1, ids.data_ptr(), dists.data_ptr())
print("perm", *st["perm"][:2])
"""
    env = dict(os.environ, PYTHONPATH=ROOT, KNNSJ_TEST_PINNED_KB="16384")
    p = subprocess.run([sys.executable, "-c", body], env=env, cwd=ROOT, timeout=300, capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-2000:]
    assert "perm 1 0" in p.stdout  # the sample's order: larger variance first
    assert "refused" not in p.stderr
