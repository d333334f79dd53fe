"""Pageable host inputs go to the device through a ring of 16 pinned pieces of 2 MB filled by several
threads: sources below and above the 8 MB line, of a whole number of pieces and of one byte row more,
and longer than the ring, dense and CSR, called in turn (a ring that still holds the last call's
pieces), have to give what the same rows on the GPU give."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mb,extra", [(7, 0), (8, 0), (10, 1), (32, 0), (75, 3)])
def test_dense_rows(mb, extra):
    import torch
    import culsh_b200 as culsh
    d = 64
    n = (mb << 20) // (4 * d) + extra
    X = np.random.default_rng(mb).standard_normal((n, d)).astype(np.float32)
    for x in (X, np.ascontiguousarray(X[::-1])):  # the second call finds the ring in use
        host = culsh.RPLSH(2, 12, seed=1).fit(x).index
        dev = culsh.RPLSH(2, 12, seed=1).fit(torch.from_numpy(x).cuda()).index
        assert np.array_equal(host.get_candidate_indices(), dev.get_candidate_indices())
        assert np.array_equal(host.get_bucket_signatures(), dev.get_bucket_signatures())


@pytest.mark.parametrize("first", [0, 5])
@pytest.mark.parametrize("nnz", [(2 << 20) - 7, (2 << 20) + 1, 19_000_001])
def test_csr_rows(nnz, first):
    import torch
    from culsh_b200._culsh_core import MinHashCore
    rng = np.random.default_rng(nnz)
    n = nnz // 100
    indptr = np.sort(rng.integers(first, nnz + 1, n + 1)).astype(np.int32)
    indptr[0], indptr[-1] = first, nnz
    indices = rng.integers(0, 1 << 20, nnz).astype(np.int32)
    core = MinHashCore(2, 2, 3)
    host = core.fit(indices, indptr, n, 1 << 20)
    dev = core.fit(torch.from_numpy(indices).cuda(), torch.from_numpy(indptr).cuda(), n, 1 << 20)
    assert np.array_equal(host.get_candidate_indices(), dev.get_candidate_indices())
    assert np.array_equal(host.get_bucket_signatures(), dev.get_bucket_signatures())
