"""A warp of the MinHash kernel takes up to sixteen rows that lie next to one another: row counts at which a warp's rows go from one
to two and to sixteen and the last warp has one or some, empty rows at the ends of a warp's rows and in runs, rows of more than one
step, ids in each of the ranges, keys with leading words and hash functions in two sweeps, against the 64-bit oracle."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,k", [(1, 2, 3), (2, 36, 8), (28_416, 8, 5), (28_417, 2, 3), (28_417, 36, 8), (28_449, 8, 5), (56_833, 36, 8),
                                   (460_001, 2, 3), (460_001, 4, 4)])
def test_rows_of_a_warp(n, L, k):
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(n + L)
    size = rng.integers(0, 6, n)
    size[rng.integers(0, n, n // 20 + 1)] = rng.integers(30, 70)
    size[np.arange(0, n, 16)[::3]] = 0
    size[np.arange(15, n, 16)[::3]] = 0
    size[n // 2:n // 2 + 40] = 0
    indptr = np.concatenate([[0], np.cumsum(size)]).astype(np.int32)
    top = np.array([1 << 10, 1 << 16, 1 << 20, 1 << 29, (1 << 31) - 1])[rng.integers(0, 5, n)]
    indices = (rng.random(indptr[-1]) * np.repeat(top, size)).astype(np.int32)
    core = core_mod.MinHashCore(L, k, 3)
    ix = core.fit(np.arange(4, dtype=np.int32), np.arange(5, dtype=np.int32), 4, (1 << 31) - 1)
    want = oracle.minhash_signatures(indices, indptr, ix.get_hash_a(), ix.get_hash_b())
    got = core.hash(indices, indptr, n, ix)
    assert np.array_equal(got.transpose(1, 0, 2).reshape(n, L * k), want)
