"""The learned radius's features from the sparse cell list (galloping over the
rows of the shells) equal those from the dense cell table, bit for bit."""
import numpy as np
import pytest

from hybrid_k_nearest_neighbor_self_join_gb300 import datasets, train_radius

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import __graft_entry__
    __graft_entry__.build_library()


@pytest.mark.parametrize("n,d", [(1_500, 1), (60_000, 1), (2_500, 2), (150_000, 2), (80_000, 3), (50_000, 4)])
def test_list_equals_dense(monkeypatch, n, d):
    x = datasets.gmm(n, d, 9, 0.2, 300 + d, dtype=np.float32)
    out = {}
    for dense in ("0", "2"):
        monkeypatch.setenv("KNNSJ_DENSE", dense)
        out[dense] = train_radius.radius_features(x, 16, 0.05)
    assert out["0"][1] == out["2"][1]
    assert np.array_equal(out["0"][0].view(np.uint32), out["2"][0].view(np.uint32))
