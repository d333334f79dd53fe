"""Lanes share a search when there are few pairs: tables of fewer, as many and more buckets than lanes search at once, queries below the first
bucket, above the last and between two, with every number of lanes and every width of a key, against the same queries in a
set large enough for a thread each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2, 4, 5, 9])  # keys of 2, 4, 8 and 16 words
@pytest.mark.parametrize("n", [1, 2, 8, 31, 32, 33, 34, 300, 5000])
def test_sets(n, k):
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(n + k)
    L, most = 9, 1000
    X = rng.integers(0, 200, (n, 3))
    Q = np.concatenate([X[rng.integers(0, n, most // 2)], rng.integers(0, 200, (most - most // 2, 3))])
    Q = Q[rng.permutation(most)]
    arrays = lambda R: (np.ascontiguousarray(R.astype(np.int32)).ravel(), (3 * np.arange(len(R) + 1)).astype(np.int32))  # noqa: E731
    core = core_mod.MinHashCore(L, k, 5)
    ix = core.fit(*arrays(X), n, 200)
    whole = core.query(*arrays(Q), most, ix)
    off, ids = whole.get_offsets().astype(np.int64), whole.get_indices()
    for nq in (1, 2, 5, 14, 15, 28, 29, 57, 113, 228, 455, 910):
        part = core.query(*arrays(Q[:nq]), nq, ix)
        assert np.array_equal(part.get_offsets().astype(np.int64), off[:nq + 1])
        assert np.array_equal(part.get_indices(), ids[:off[nq]])


@pytest.mark.parametrize("n,k", [(40, 8), (3000, 12), (3000, 32), (3000, 50)])  # keys of one and two words
def test_signs(n, k):
    import culsh_b200 as culsh
    rng = np.random.default_rng(k)
    X = rng.standard_normal((n, 16)).astype(np.float32)
    Q = np.concatenate([X[rng.integers(0, n, 300)], rng.standard_normal((700, 16))]).astype(np.float32)[rng.permutation(1000)]
    m = culsh.RPLSH(10, k, seed=2).fit(X)
    whole = m.query(Q)
    off, ids = whole.get_offsets().astype(np.int64), whole.get_indices()
    for nq in (1, 3, 12, 13, 25, 26, 51, 102, 204, 409, 819):
        part = m.query(Q[:nq])
        assert np.array_equal(part.get_offsets().astype(np.int64), off[:nq + 1])
        assert np.array_equal(part.get_indices(), ids[:off[nq]])
