"""Small fits and small sets of queries go on before the host has seen their counts, and what was launched is done again
where the counts ask for something else: hash values that span more than the compressed sort takes, in tables
that one CTA sorts (bucket arrays below and above the 4 MB that are made beforehand); sets of up to 4,096 queries with more
ids than fit, with sets for the windows, and on an index with a sort path; each against the same queries in a
larger set."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b):
    for f in ("get_indices", "get_offsets", "get_counts"):
        assert np.array_equal(getattr(a, f)(), getattr(b, f)())


@pytest.mark.parametrize("n,L", [(1, 2), (5, 8), (1000, 8), (8192, 3), (12_288, 40), (12_288, 2)])
@pytest.mark.parametrize("scale", [0.2, 2.0, 4.4, 9.0, 200.0])
def test_p_stable_spans(n, L, scale):
    import culsh_b200 as culsh
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(n)
    d, k = 8, 8
    base = (scale * rng.standard_normal((n // 3 + 1, d))).astype(np.float32)
    X = base[rng.integers(0, len(base), n)]
    core = core_mod.PSLSHCore(L, k, 1, 3)
    ix = core.fit_float(X, n, d)
    sig = core.hash(X, ix)
    cand, tab, off = ix.get_candidate_indices(), ix.get_table_bucket_offsets(), ix.get_bucket_candidate_offsets()
    keys = ix.get_bucket_signatures().reshape(ix.n_total_buckets, -1)
    assert len(off) == ix.n_total_buckets + 1 and off[-1] == n * L
    for t in range(L):
        raw = np.ascontiguousarray(sig[t]).view(np.uint8).reshape(n, 4 * k)
        order = np.lexsort(tuple(raw[:, j] for j in range(4 * k - 1, -1, -1)))
        assert np.array_equal(cand[t * n:(t + 1) * n], order)
        srt = raw[order]
        head = np.concatenate([[True], (srt[1:] != srt[:-1]).any(axis=1)])
        assert np.array_equal(keys[tab[t]:tab[t + 1]], srt[head])
    lsh = culsh.PStableLSH(L, k, window_size=1, seed=3)
    _same(lsh.fit_query(X), lsh.fit(X).query(X))


@pytest.mark.parametrize("n,L,k", [(60_000, 4, 2), (60_000, 4, 6), (60_000, 12, 12), (2_400_000, 4, 12)])
def test_queries_equal_those_of_a_larger_set(n, L, k):
    import culsh_b200 as culsh
    rng = np.random.default_rng(k)
    X = rng.standard_normal((n, 6)).astype(np.float32)
    Q = np.concatenate([X[:2000], rng.standard_normal((2200, 6)), 1e4 * np.eye(6)]).astype(np.float32)
    if k == 2:
        Q = np.concatenate([Q[:30], Q[4195:]])
    m = culsh.RPLSH(L, k, seed=6).fit(X)
    big = np.concatenate([Q, Q[:max(1, 4200 - len(Q))]]) if k != 2 else Q
    whole = m.query(big)
    off, ids = whole.get_offsets().astype(np.int64), whole.get_indices()
    for a, b in [(0, 1), (0, 2), (3, 40), (0, 3000), (100, 4196), (len(Q) - 6, len(Q))]:
        a, b = min(a, len(Q) - 1), min(b, len(Q))
        part = m.query(Q[a:b])
        assert np.array_equal(part.get_offsets().astype(np.int64), off[a:b + 1] - off[a])
        assert np.array_equal(part.get_indices(), ids[off[a]:off[b]])


def test_windows_launched_ahead_are_timed():
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(4)
    n, d = 60_000, 6
    X = rng.standard_normal((n, d)).astype(np.float32)
    core = core_mod.RPLSHCore(4, 2, 6)
    core.set_profiling(True)
    try:
        ix = core.fit_float(X, n, d)
        for nq in (1, 30, 200):  # the last is too many for windows before the counts are known
            assert core.query_float(X[:nq], nq, ix).n_total_candidates > 1024 * nq
            assert core.last_stats()["dedupe_ms"] > 0
    finally:
        core.set_profiling(False)


def test_small_sets_are_gathered_once():
    """Next to sets for the windows that wait for their counts, the small ones that were gathered ahead stay as they are."""
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(5)
    n, d = 60_000, 32
    X = rng.standard_normal((n, d)).astype(np.float32)
    X[:3000] = X[0]
    core = core_mod.RPLSHCore(4, 16, 6)
    ix = core.fit_float(X, n, d)
    few = np.ascontiguousarray(X[10_000:10_100])
    mixed = few.copy()
    mixed[::10] = X[0]
    small = core.query_float(few, 100, ix)
    launches = core.last_stats()["launches"]
    assert int(small.get_counts().max()) < 256
    got = core.query_float(mixed, 100, ix)
    # the windows and the copy of the pieces
    assert core.last_stats()["launches"] == launches + 2
    counts = got.get_counts()
    assert (counts[::10] >= 3000).all()
    for q in (1, 10, 55):
        one = core.query_float(mixed[q:q + 1], 1, ix)
        off = got.get_offsets()
        assert np.array_equal(one.get_indices(), got.get_indices()[int(off[q]):int(off[q + 1])])
