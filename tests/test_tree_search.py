"""The box-tree search against an exact brute force, at the sizes where it can
go wrong: partly filled leaves, blocks and levels of the tree, every compiled
dimension count and the runtime one, selection buffers of every kind, both
data types with and without the float screen, exact ties, far outliers."""
import numpy as np
import pytest

import oracle
import hybrid_k_nearest_neighbor_self_join_gb300 as kj
from hybrid_k_nearest_neighbor_self_join_gb300 import datasets

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import __graft_entry__
    __graft_entry__.build_library()
    __graft_entry__.build_oracle()


def check(monkeypatch, x, k, queries=None, **kw):
    monkeypatch.setenv("KNNSJ_TREE", "2")  # at every dimension count
    ids, dists = kj.selfjoin(x, k, **kw)
    perm, _ = kj.reorder_dims(x)
    n = x.shape[0]
    q = np.arange(n) if n <= 3000 else np.unique(np.random.default_rng(0).integers(0, n, 1500))
    if queries is not None:
        q = np.union1d(q, queries)
    bi, bd = oracle.bruteforce(np.ascontiguousarray(x[:, perm]), k + 1, q.astype(np.uint32))
    ub = np.uint32 if x.dtype == np.float32 else np.uint64
    assert np.array_equal(ids[q], bi)
    assert np.array_equal(dists[q].view(ub), bd.view(ub))


@pytest.mark.parametrize("n", [2, 31, 32, 33, 1023, 1024, 1025, 2049, 32767, 32769, 33000])
@pytest.mark.parametrize("d,dtype", [(2, np.float32), (4, np.float32), (6, np.float64)])
def test_sizes(monkeypatch, n, d, dtype):
    x = datasets.gmm(n, d, 5, 0.2, n + d, dtype=dtype)
    check(monkeypatch, x, min(8, n - 1))
    check(monkeypatch, x, min(8, n - 1), radius_mode=kj.RADIUS_LEARNED)


@pytest.mark.parametrize("d", [1, 2, 3, 4, 5, 6, 7, 8, 9, 12, 17, 40])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_dimensions(monkeypatch, d, dtype):
    x = datasets.gmm(5_003, d, 7, 0.1, 50 + d, dtype=dtype)
    check(monkeypatch, x, 15)


@pytest.mark.parametrize("k", [1, 31, 47, 48, 95, 191, 223, 224, 300, 1000])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_row_lengths(monkeypatch, k, dtype):
    x = datasets.gmm(4_001, 4, 6, 0.2, 70 + k, dtype=dtype)
    check(monkeypatch, x, k)


@pytest.mark.parametrize("mode", [kj.RADIUS_PLAIN, kj.RADIUS_LEARNED])
def test_exact_ties(monkeypatch, mode):
    base = datasets.uniform(500, 4, 9)
    x = np.ascontiguousarray(np.repeat(base, 40, axis=0)[np.random.default_rng(1).permutation(20_000)])
    check(monkeypatch, x, 24, radius_mode=mode)
    check(monkeypatch, x.astype(np.float64), 24, radius_mode=mode)


@pytest.mark.parametrize("screen", ["0", "1"])
@pytest.mark.parametrize("offset", [0.0, 1e4, 1e12])
def test_double_screen(monkeypatch, screen, offset):
    # a large offset leaves few float bits for the differences; without the
    # screen every distance is taken in double
    monkeypatch.setenv("KNNSJ_FLOAT_PREFILTER", screen)
    x = datasets.gmm(6_000, 5, 6, 0.2, 33, dtype=np.float64) * 1e-2 + offset
    check(monkeypatch, x, 12)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_far_outliers_and_clumps(monkeypatch, dtype):
    rng = np.random.default_rng(2)
    c = rng.normal(0.0, 1e-3, (12_000, 3))
    far = rng.uniform(-1.0, 1.0, (9, 3)) * 20.0
    x = np.concatenate([c, c[:4_000] * 1e-2 + 0.5, far]).astype(dtype)
    check(monkeypatch, x, 16, queries=np.arange(16_000, 16_009))


@pytest.mark.parametrize("d,dtype,mode", [(8, np.float64, kj.RADIUS_LEARNED), (8, np.float64, kj.RADIUS_PLAIN),
                                          (2, np.float64, kj.RADIUS_PLAIN), (3, np.float32, kj.RADIUS_LEARNED)])
def test_fixed_scratch_at_its_limits(d, dtype, mode):
    # the largest problem of the fixed scratch array: grid, tree and radii all
    # come from it
    torch = pytest.importorskip("torch")
    import ctypes
    from hybrid_k_nearest_neighbor_self_join_gb300 import _lib
    n, k = 65_536, 127
    x = datasets.gmm(n, d, 9, 0.3, 60 + d, dtype=dtype)
    dev = torch.from_numpy(x).cuda()
    ids = [torch.full((n, k + 1), -7, dtype=torch.int32, device="cuda") for _ in range(2)]
    dists = [torch.full((n, k + 1), -1.0, dtype=dev.dtype, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    opts = _lib.Options.make(radius_mode=mode)
    code = _lib.KNNSJ_F32 if dtype == np.float32 else _lib.KNNSJ_F64
    args = [ctypes.c_void_p(dev.data_ptr()), code, n, d, k, ctypes.byref(opts)]
    lib = _lib.load()
    _lib.check(lib.knnsj_selfjoin_device_noalloc(*args, ctypes.c_void_p(ids[0].data_ptr()),
                                                 ctypes.c_void_p(dists[0].data_ptr())))
    st = _lib.Stats.make()
    _lib.check(lib.knnsj_selfjoin_device(*args, ctypes.c_void_p(ids[1].data_ptr()),
                                         ctypes.c_void_p(dists[1].data_ptr()), ctypes.byref(st)))
    assert torch.equal(ids[0], ids[1]) and torch.equal(dists[0], dists[1])
