"""Large candidate sets of indexes with more than 256 tables are merged by a CTA for each query, with a bitmap of a window of the rows after the other and,
above 1,024 tables, the tables in groups: sets of no id to nearly all rows, one window and several, rows at the edges of windows, and a
self-join, against the signatures by brute force."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _keys(sig):
    """[L][n][k] sign bytes -> [n][L] numbers."""
    return (sig.astype(np.int64) << np.arange(sig.shape[2])).sum(axis=2).T.copy()


def _rows(n, d, rng):
    X = rng.standard_normal((n, d)).astype(np.float32)
    X[rng.permutation(n)[:1300]] = X[7]  # alike, so that they are in one another's lists of all tables
    for e in range(4096, n, 4096):
        X[e - 1:e + 1] = X[8]
    X[n - 1] = X[8]
    return X


@pytest.mark.parametrize("bits", [None, 4096, 8192, 20_480])
@pytest.mark.parametrize("L,n,k", [(257, 20_000, 6), (257, 4096, 3), (1024, 9000, 5), (1025, 9000, 9), (1025, 20_481, 3), (2100, 8193, 8)])
def test_queries(L, n, k, bits, monkeypatch):
    import culsh_b200 as culsh
    from culsh_b200 import _culsh_core as core_mod
    if bits:
        monkeypatch.setenv("CULSH_BITMAP_BITS", str(bits))
    rng = np.random.default_rng(L + n)
    d = 6
    X = _rows(n, d, rng)
    Q = np.concatenate([X[7:9], X[:2] * 3, rng.standard_normal((3, d)), -X[7:8]]).astype(np.float32)
    m = culsh.RPLSH(L, k, seed=3).fit(X)
    core = core_mod.RPLSHCore(L, k, 3)
    x, q = _keys(core.hash(X, m.index)), _keys(core.hash(Q, m.index))
    want = [np.flatnonzero((x == row).any(axis=1)) for row in q]
    raw = [int((x == row).sum()) for row in q]
    assert max(raw) > 300_000 and max(map(len, want)) > 1300
    got = m.query(Q)
    assert np.array_equal(got.get_counts(), [len(w) for w in want])
    assert np.array_equal(got.get_indices(), np.concatenate(want))


@pytest.mark.parametrize("bits", [None, 4096])
@pytest.mark.parametrize("L,n,k", [(257, 6000, 6), (1025, 5000, 9)])
def test_self_join(L, n, k, bits, monkeypatch):
    import culsh_b200 as culsh
    from culsh_b200 import _culsh_core as core_mod
    if bits:
        monkeypatch.setenv("CULSH_BITMAP_BITS", str(bits))
    rng = np.random.default_rng(L)
    X = _rows(n, 6, rng)
    lsh = culsh.RPLSH(L, k, seed=2)
    x = _keys(core_mod.RPLSHCore(L, k, 2).hash(X, lsh.fit(X).index))
    got = lsh.fit_query(X)
    offsets, ids = got.get_offsets().astype(np.int64), got.get_indices()
    assert len(offsets) == n + 1 and offsets[-1] == len(ids)
    for row in [0, 7, 8, 4095, 4096, n - 1, *rng.integers(0, n, 30)]:
        assert np.array_equal(ids[offsets[row]:offsets[row + 1]], np.flatnonzero((x == x[row]).any(axis=1)))
