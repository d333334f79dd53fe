"""The self-join takes its bucket lists from the finished buckets, packed into one word per (row,
table), and the query path looks them up by key: both have to give the same CSR.  Sizes at the
edges of the 2048-item tiles of the bucket pass, with blocks of equal rows that make buckets of one,
two and many rows, across a tile, and (n = 1,100,000: 21 position bits, 10 for the number of rows)
longer than the packed word can say."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,k,copies", [
    (1, 2, 8, []), (2, 2, 8, [2]), (2047, 3, 20, [2, 3]), (2048, 3, 20, [4, 5]), (2049, 65, 20, [2, 130]),
    (4097, 129, 20, [1025, 33]), (30_000, 4, 22, [1400, 2, 2, 2]), (1_100_000, 2, 30, [1500, 3, 2]),
])
def test_self_join_equals_query_with_own_rows(n, L, k, copies):
    import culsh_b200 as culsh
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, 12)).astype(np.float32)
    at = rng.permutation(n)
    i = 0
    for c in copies:  # c equal rows at scattered places
        X[at[i:i + c]] = X[at[i]]
        i += c
    lsh = culsh.RPLSH(L, k, seed=4)
    want = lsh.fit(X).query(X)
    got = lsh.fit_query(X)
    assert np.array_equal(got.get_offsets(), want.get_offsets())
    assert np.array_equal(got.get_indices(), want.get_indices())
    assert np.array_equal(got.get_counts(), want.get_counts())
