"""Pageable host inputs of 32 MB and more go to the device through a ring of 8 pinned pieces of 2 MB filled by
several threads, once a handle has been given 160 MB: sources below and above the 32 MB line, of a whole
number of pieces and of one byte row more, and longer than the ring, dense and CSR, called in turn (a
ring that still holds the last call's pieces), before there is a ring and with it, have to give what the
same rows on the GPU give."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ring(wanted):
    """A handle without a ring, or with one."""
    import culsh_b200 as culsh
    from culsh_b200 import _culsh_core as core_mod
    core_mod.RPLSHCore(1, 2, 1).trim_scratch(0)
    if wanted:
        culsh.RPLSH(1, 2, seed=1).fit(np.ones((1 << 20, 40), np.float32))  # 160 MB


@pytest.mark.parametrize("ring", [False, True])
@pytest.mark.parametrize("mb,extra", [(31, 0), (32, 0), (33, 1), (75, 3), (165, 1), (260, 1)])
def test_dense_rows(mb, extra, ring):
    import torch
    import culsh_b200 as culsh
    d = 64
    n = (mb << 20) // (4 * d) + extra
    X = np.random.default_rng(mb).standard_normal((n, d), dtype=np.float32)
    _ring(ring)
    for x in (X, np.ascontiguousarray(X[::-1])):  # the second call finds the ring in use
        host = culsh.RPLSH(2, 12, seed=1).fit(x).index
        dev = culsh.RPLSH(2, 12, seed=1).fit(torch.from_numpy(x).cuda()).index
        assert np.array_equal(host.get_candidate_indices(), dev.get_candidate_indices())
        assert np.array_equal(host.get_bucket_signatures(), dev.get_bucket_signatures())


@pytest.mark.parametrize("first", [0, 5])
@pytest.mark.parametrize("nnz", [(8 << 20) - 7, (8 << 20) + 1, 19_000_001])
def test_csr_rows(nnz, first):
    import torch
    from culsh_b200._culsh_core import MinHashCore
    rng = np.random.default_rng(nnz)
    n = nnz // 100
    indptr = np.sort(rng.integers(first, nnz + 1, n + 1)).astype(np.int32)
    indptr[0], indptr[-1] = first, nnz
    indices = rng.integers(0, 1 << 20, nnz).astype(np.int32)
    core = MinHashCore(2, 2, 3)
    _ring(True)
    host = core.fit(indices, indptr, n, 1 << 20)
    dev = core.fit(torch.from_numpy(indices).cuda(), torch.from_numpy(indptr).cuda(), n, 1 << 20)
    assert np.array_equal(host.get_candidate_indices(), dev.get_candidate_indices())
    assert np.array_equal(host.get_bucket_signatures(), dev.get_bucket_signatures())
