"""In-degrees of a table in which one id stands more than 2^32 times."""
import pytest

import hybrid_k_nearest_neighbor_self_join_gb300 as kj

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def built():
    import __graft_entry__
    __graft_entry__.build_library()


def test_one_id_everywhere():
    n = K = 65_540  # n K = 2^32 + 524 304
    if torch.cuda.mem_get_info()[0] < 48 << 30:
        pytest.skip("the table takes 34 GB")
    ids = torch.full((n, K), 7, dtype=torch.int32, device="cuda")
    dists = torch.zeros((n, K), dtype=torch.float32, device="cuda")
    mean = torch.empty(n, dtype=torch.float64, device="cuda")
    dist_rank, degree_rank = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    degree = torch.empty(n, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    kj.outlier_scores_device(ids.data_ptr(), dists.data_ptr(), "float32", n, K, mean.data_ptr(), dist_rank.data_ptr(),
                             degree.data_ptr(), degree_rank.data_ptr())
    torch.cuda.synchronize()
    want = torch.zeros(n, dtype=torch.int64, device="cuda")
    want[7] = n * K
    assert torch.equal(degree, want)
    rank = torch.arange(n, dtype=torch.int32, device="cuda")
    rank[7] = n - 1
    rank[8:] -= 1
    assert torch.equal(degree_rank, rank)
    del ids, dists
    torch.cuda.empty_cache()
