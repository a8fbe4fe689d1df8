"""Which joins the box tree takes, and that it answers them.

A join's path is told by its lines at KNNSJ_VERBOSE=2; its rows are compared
with brute force.
"""
import ctypes

import numpy as np
import pytest

import oracle
import hybrid_k_nearest_neighbor_self_join_gb300 as kj
from hybrid_k_nearest_neighbor_self_join_gb300 import _lib, datasets

pytestmark = pytest.mark.gpu

F, D = np.float32, np.float64
PLAIN, LEARNED = kj.RADIUS_PLAIN, kj.RADIUS_LEARNED


@pytest.fixture(scope="module", autouse=True)
def built():
    import __graft_entry__
    __graft_entry__.build_library()
    __graft_entry__.build_oracle()


def check_brute(x, ids, dists, queries):
    perm, _ = kj.reorder_dims(x)
    bi, bd = oracle.bruteforce(np.ascontiguousarray(x[:, perm]), ids.shape[1], queries.astype(np.uint32))
    ub = np.uint32 if x.dtype == np.float32 else np.uint64
    assert np.array_equal(ids[queries], bi)
    assert np.array_equal(dists[queries].view(ub), bd.view(ub))


@pytest.mark.parametrize("tree,d,dtype,k,mode,env,kw", [
    # uniform radii, and learned ones in three and more dimensions
    (True, 1, F, 8, PLAIN, {}, {}),
    (True, 2, F, 8, PLAIN, {}, {}),
    (True, 2, D, 8, PLAIN, {}, {}),
    (True, 3, F, 8, LEARNED, {}, {}),
    (True, 5, D, 8, LEARNED, {}, {}),
    (True, 12, F, 8, PLAIN, {}, {}),
    (True, 40, D, 8, PLAIN, {}, {}),
    # learned radii in one and two dimensions: query tiles and rings
    (False, 1, F, 8, LEARNED, {}, {}),
    (False, 2, F, 8, LEARNED, {}, {}),
    (False, 2, D, 8, LEARNED, {}, {}),
    # the longest rows
    (True, 4, F, 223, PLAIN, {}, {}),
    (False, 4, F, 224, PLAIN, {}, {}),
    (True, 4, D, 191, PLAIN, {}, {}),
    (False, 4, D, 192, PLAIN, {}, {}),
    # a cap on the schedule's passes, the switches
    (False, 3, F, 8, PLAIN, {}, {"max_iterations": 5000}),
    (False, 3, F, 8, PLAIN, {"KNNSJ_TREE": "0"}, {}),
    (True, 2, D, 8, LEARNED, {"KNNSJ_TREE": "2"}, {}),
    (False, 3, F, 8, LEARNED, {"KNNSJ_TILE": "3"}, {}),
    (False, 4, D, 8, PLAIN, {"KNNSJ_FLOAT_PREFILTER": "0"}, {}),
])
def test_path(monkeypatch, capfd, tree, d, dtype, k, mode, env, kw):
    n = 5_003
    x = datasets.gmm(n, d, 7, 0.1, 700 + d, dtype=dtype)
    for name in ("KNNSJ_TREE", "KNNSJ_TILE"):
        monkeypatch.delenv(name, raising=False)
    for name, v in env.items():
        monkeypatch.setenv(name, v)
    monkeypatch.setenv("KNNSJ_VERBOSE", "2")
    capfd.readouterr()
    ids, dists = kj.selfjoin(x, k, radius_mode=mode, **kw)
    assert ("box tree" in capfd.readouterr().err) == tree
    check_brute(x, ids, dists, np.arange(0, n, 13))


@pytest.mark.parametrize("scale,tree", [(1e16, True), (1e18, False)])
def test_coordinates_beyond_the_float_screen(monkeypatch, capfd, scale, tree):
    x = datasets.gmm(5_003, 4, 7, 0.1, 704, dtype=D) * scale
    monkeypatch.setenv("KNNSJ_VERBOSE", "2")
    capfd.readouterr()
    ids, dists = kj.selfjoin(x, 8)
    assert ("box tree" in capfd.readouterr().err) == tree
    check_brute(x, ids, dists, np.arange(0, 5_003, 13))


@pytest.mark.parametrize("d,dtype,mode", [(8, D, LEARNED), (8, F, PLAIN), (2, D, PLAIN)])
def test_fixed_scratch(monkeypatch, capfd, d, dtype, mode):
    # the largest problem of the fixed scratch array, through the tree, against
    # brute force
    torch = pytest.importorskip("torch")
    n, k = 65_536, 127
    x = datasets.gmm(n, d, 9, 0.3, 60 + d, dtype=dtype)
    dev = torch.from_numpy(x).cuda()
    ids = torch.full((n, k + 1), -7, dtype=torch.int32, device="cuda")
    dists = torch.full((n, k + 1), -1.0, dtype=dev.dtype, device="cuda")
    torch.cuda.synchronize()
    monkeypatch.setenv("KNNSJ_VERBOSE", "2")
    capfd.readouterr()
    opts = _lib.Options.make(radius_mode=mode)
    _lib.check(_lib.load().knnsj_selfjoin_device_noalloc(
        ctypes.c_void_p(dev.data_ptr()), _lib.KNNSJ_F32 if dtype == F else _lib.KNNSJ_F64, n, d, k, ctypes.byref(opts),
        ctypes.c_void_p(ids.data_ptr()), ctypes.c_void_p(dists.data_ptr())))
    torch.cuda.synchronize()
    assert "box tree" in capfd.readouterr().err
    check_brute(x, ids.cpu().numpy(), dists.cpu().numpy(), np.arange(0, n, 2_311))


def test_large_learned_3d_by_density(monkeypatch, capfd):
    # evenly filled space stays with the query tiles from a million points on,
    # uneven density goes through the tree; fewer points always
    rng = np.random.default_rng(7)
    monkeypatch.setenv("KNNSJ_VERBOSE", "2")
    for x, tree in ((rng.random((1_000_000, 3)), False), (datasets.gmm(1_000_000, 3, 12, 0.2, 8), True),
                    (rng.random((999_999, 3)), True)):
        x = x.astype(F)
        capfd.readouterr()
        ids, dists, st = kj.selfjoin(x, 8, radius_mode=LEARNED, return_stats=True)
        assert ("box tree" in capfd.readouterr().err) == tree
        check_brute(x, ids, dists, np.arange(0, len(x), 20_011))
        perm = st["perm"][:3]
        lo, width = x[:, perm].min(0), F(st["eps0"])
        cells = np.unique(((x[:, perm] - lo) / width).astype(np.int64) @ np.array([1, 1 << 20, 1 << 40]))
        assert abs(st["nonempty_cells"] - len(cells)) <= len(cells) * 1e-3
