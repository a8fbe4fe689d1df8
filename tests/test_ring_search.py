"""The grid's ring search where the box tree would answer by itself.

The ring search with its retry graph, grid rebuilds and exact tail still takes
long rows, joins with a cap on the passes, streamed rows and two-dimensional
learned joins.  KNNSJ_TREE=0 sends every join to it; each test checks a figure
that a box-tree join (three passes at most, one index rebuild) cannot have.
"""
import ctypes

import numpy as np
import pytest

import oracle
import hybrid_k_nearest_neighbor_self_join_gb300 as kj
from hybrid_k_nearest_neighbor_self_join_gb300 import _lib, datasets

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import __graft_entry__
    __graft_entry__.build_library()
    __graft_entry__.build_oracle()


@pytest.fixture(autouse=True)
def ring(monkeypatch):
    monkeypatch.setenv("KNNSJ_TREE", "0")


def bits(a):
    return a.view(np.uint32 if a.dtype == np.float32 else np.uint64)


def same_rows(a, b):
    assert np.array_equal(a[0], b[0])
    assert np.array_equal(bits(a[1]), bits(b[1]))


def check_brute(x, ids, dists, queries):
    perm, _ = kj.reorder_dims(x)
    same_rows((ids[queries], dists[queries]),
              oracle.bruteforce(np.ascontiguousarray(x[:, perm]), ids.shape[1], queries.astype(np.uint32)))


@pytest.mark.parametrize("mode,offset", [(kj.RADIUS_PLAIN, 0.0), (kj.RADIUS_LEARNED, -1.0)])
def test_graph_passes_match_host_passes(monkeypatch, mode, offset):
    x = datasets.gmm(120_000, 4, 30, 0.2, 21, dtype=np.float32)
    out = {}
    for g in ("0", "1"):
        monkeypatch.setenv("KNNSJ_GRAPH", g)
        out[g] = kj.selfjoin(x, 32, beta=0.0, radius_mode=mode, radius_offset=offset, return_stats=True)
    same_rows(out["0"], out["1"])
    a, b = out["0"][2], out["1"][2]
    assert a["iterations"] > 3
    for key in ("iterations", "regrids", "candidates", "queries_run", "eps_final"):
        assert a[key] == b[key], key
    check_brute(x, *out["1"][:2], np.arange(0, 120_000, 911))


def test_dense_and_sparse_cell_lookup_agree(monkeypatch):
    x = datasets.sky_like(60_000, seed=13)
    out = {}
    for dense in ("0", "2"):
        monkeypatch.setenv("KNNSJ_DENSE", dense)
        out[dense] = kj.selfjoin(x, 16, beta=0.025, return_stats=True)
        assert out[dense][2]["iterations"] > 3
    same_rows(out["0"], out["2"])
    check_brute(x, *out["0"][:2], np.arange(0, 60_000, 499))


def test_far_outliers(monkeypatch):
    # tail 0: the grid is rebuilt for the outliers' radii; 1: the last few
    # queries are finished by a scan over all points
    rng = np.random.default_rng(23)
    c = rng.normal(0.0, 0.01, (40_000, 6)).astype(np.float32)
    o = rng.uniform(-1.0, 1.0, (12, 6)).astype(np.float32)
    x = np.concatenate([c, o])
    q = np.concatenate([np.arange(40_000, 40_012), np.arange(0, 40_000, 997)])
    out = {}
    for tail in ("0", "1"):
        monkeypatch.setenv("KNNSJ_TAIL_BRUTE", tail)
        out[tail] = kj.selfjoin(x, 16, beta=0.05, radius_mode=kj.RADIUS_LEARNED, return_stats=True)
        check_brute(x, *out[tail][:2], q)
        assert out[tail][2]["iterations"] > 3 and out[tail][2]["regrids"] > 1
    same_rows(out["0"], out["1"])


@pytest.mark.parametrize("dtype,mode", [(np.float32, kj.RADIUS_PLAIN), (np.float64, kj.RADIUS_PLAIN),
                                        (np.float64, kj.RADIUS_LEARNED)])
def test_sparse_tail_matches_rebuilt_grids(monkeypatch, dtype, mode):
    rng = np.random.default_rng(24)
    c = (rng.normal(0.0, 0.002, (60_000, 2)) + rng.integers(0, 4, (60_000, 1)) * 0.01).astype(dtype)
    x = np.concatenate([c, rng.uniform(-1.0, 1.0, (7, 2)).astype(dtype)])
    out = {}
    for tail in ("0", "2"):
        monkeypatch.setenv("KNNSJ_TAIL_BRUTE", tail)
        out[tail] = kj.selfjoin(x, 24, beta=0.0, radius_mode=mode, return_stats=True)
    same_rows(out["0"], out["2"])
    assert out["0"][2]["iterations"] > 3
    assert out["0"][2]["regrids"] > out["2"][2]["regrids"]  # 2: forced at the first due rebuild
    check_brute(x, *out["2"][:2], np.arange(60_000, 60_007))


@pytest.mark.parametrize("offset", [0.0, 3.0e5])
def test_double_float_screen_bound(monkeypatch, offset):
    # far from the origin the float screen lets every candidate through, near it
    # rejects most
    x = datasets.gmm(30_000, 4, 8, 0.2, 22, dtype=np.float64) * 1e-3 + offset
    ids, dists, st = kj.selfjoin(x, 12, num_indexed_dims=4, beta=0.05, return_stats=True)
    rc, oids, odists, ost = oracle.join(x, 12, di=4, beta=0.05)
    assert rc == 0 and st["eps0"] == ost.eps0 and st["iterations"] > 3
    same_rows((ids, dists), (oids, odists))
    monkeypatch.setenv("KNNSJ_FLOAT_PREFILTER", "0")
    same_rows((ids, dists), kj.selfjoin(x, 12, num_indexed_dims=4, beta=0.05))


def test_pass_cap_takes_the_ring_search(monkeypatch):
    x = datasets.gmm(30_000, 3, 8, 0.2, 25, dtype=np.float32)
    monkeypatch.setenv("KNNSJ_TREE", "1")
    ids, dists, st = kj.selfjoin(x, 12, max_iterations=5000, return_stats=True)
    assert st["iterations"] > 3
    same_rows((ids, dists), kj.selfjoin(x, 12))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_fixed_scratch_holds_rebuilt_grids(dtype):
    # the largest problem of the fixed scratch array: the schedule widens the
    # radius until the grid is rebuilt, and every rebuilt buffer fits
    torch = pytest.importorskip("torch")
    n, d, k = 65_536, 8, 127
    x = datasets.gmm(n, d, 6, 0.05, 13, dtype=dtype)
    dev = torch.from_numpy(x).cuda()
    ids = [torch.full((n, k + 1), -7, dtype=torch.int32, device="cuda") for _ in range(2)]
    dists = [torch.full((n, k + 1), -1.0, dtype=dev.dtype, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    opts = _lib.Options.make(beta=0.0)
    code = _lib.KNNSJ_F32 if dtype == np.float32 else _lib.KNNSJ_F64
    args = [ctypes.c_void_p(dev.data_ptr()), code, n, d, k, ctypes.byref(opts)]
    lib = _lib.load()
    _lib.check(lib.knnsj_selfjoin_device_noalloc(*args, ctypes.c_void_p(ids[0].data_ptr()),
                                                 ctypes.c_void_p(dists[0].data_ptr())))
    st = _lib.Stats.make()
    _lib.check(lib.knnsj_selfjoin_device(*args, ctypes.c_void_p(ids[1].data_ptr()),
                                         ctypes.c_void_p(dists[1].data_ptr()), ctypes.byref(st)))
    assert st.regrids >= 1 and st.iterations > 3, (st.regrids, st.iterations)
    assert torch.equal(ids[0], ids[1]) and torch.equal(dists[0], dists[1])
    check_brute(x, ids[0].cpu().numpy(), dists[0].cpu().numpy(), np.arange(0, n, 2_311))
