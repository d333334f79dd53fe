"""Up to 2,048 (table, query) pairs are looked up, counted and scanned by one CTA: query counts on both
sides of its 1024 threads and of that line have to give what the same queries give in a large set, for
lists that are empty, short, and long enough for each of the gather's paths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,k", [(1, 12), (2, 3), (2, 14), (32, 16), (33, 5), (2048, 8)])
def test_equals_the_large_set(L, k):
    import culsh_b200 as culsh
    rng = np.random.default_rng(L)
    X = rng.standard_normal((30_000, 10)).astype(np.float32)
    Q = rng.standard_normal((2100, 10)).astype(np.float32)
    Q[::3] = X[:700]
    n_all = min(2100, max(70, 300_000 // L))
    m = culsh.RPLSH(L, k, seed=8).fit(X)
    whole = m.query(Q[:n_all])
    off, ids = whole.get_offsets().astype(np.int64), whole.get_indices()
    for nq in sorted({1, 2, 63, 64, 65, 1023, 1024, 1025, 2048, 2049, 2048 // L, 2048 // L + 1}):
        if not 0 < nq <= n_all:
            continue
        part = m.query(Q[:nq])
        assert np.array_equal(part.get_offsets().astype(np.int64), off[:nq + 1])
        assert np.array_equal(part.get_indices(), ids[:off[nq]])


def test_no_list_at_all():
    import culsh_b200 as culsh
    X = np.ones((50, 8), np.float32)
    m = culsh.RPLSH(3, 40, seed=8).fit(X)
    c = m.query(-X[:5])
    assert c.n_total_candidates == 0 and not c.get_offsets().any()
