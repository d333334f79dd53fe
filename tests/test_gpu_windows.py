"""Large candidate sets are merged by a CTA for each (query, window of the rows): sets of a few ids to many thousands in a
window and of none at all, ids at the edges of windows and of their 32- and 128-bit groups, every id in several lists, a
self-join whose own row is before, in and behind a window, and results brought together inside their raw array."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lists(model, X_sig, Q_sig, n, L):
    """Candidates of every query by brute force over the signatures [n][L][k]."""
    out = []
    for q in Q_sig:
        hit = (X_sig == q[None]).all(axis=2).any(axis=1)
        out.append(np.flatnonzero(hit).astype(np.int32))
    return out


def _assert_lists(cand, want):
    off = cand.get_offsets().astype(np.int64)
    assert np.array_equal(np.diff(off), [len(w) for w in want])
    assert np.array_equal(cand.get_indices(), np.concatenate(want))


@pytest.mark.parametrize("bits", [None, 4096, 8192, 20_480, 65_536])
@pytest.mark.parametrize("slices", [0, 1])
def test_set_sizes_and_edges(bits, slices, monkeypatch):
    import culsh_b200 as culsh
    from culsh_b200 import _culsh_core as core_mod
    n, d, L, k = 65_537, 6, 3, 9
    if bits:
        monkeypatch.setenv("CULSH_CHAIN_BITS", str(bits))
    monkeypatch.setenv("CULSH_CHAIN_SLICES", str(slices))
    rng = np.random.default_rng(1)
    X = rng.standard_normal((n, d)).astype(np.float32)
    proto = rng.standard_normal((8, d)).astype(np.float32)
    # groups of equal rows: every one of them is in all lists of its prototype
    at = 0
    perm = rng.permutation(n)
    for j, size in enumerate([1025, 4095, 4096, 4097, 9000]):
        X[perm[at:at + size]] = proto[j]
        at += size
    for e in range(0, n, 4096):  # rows at the edges of windows and groups
        for r in (e - 1, e, e + 1, e + 31, e + 32, e + 127, e + 128):
            if 0 <= r < n:
                X[r] = proto[5]
    X[40_000:42_000] = proto[6]   # inside one window or two
    X[:1500] = proto[7]
    Q = np.concatenate([proto, rng.standard_normal((3, d)).astype(np.float32), -proto[:2]])
    core = core_mod.RPLSHCore(L, k, 3)
    m = culsh.RPLSH(L, k, seed=3).fit(X)
    sig = lambda Y: core.hash(Y, m.index).transpose(1, 0, 2)  # noqa: E731
    want = _lists(m, sig(X), sig(Q), n, L)
    assert max(len(w) for w in want) > 9000
    _assert_lists(m.query(Q), want)
    for q in range(len(Q)):  # one query: its window CTAs are launched before the counts are known
        _assert_lists(m.query(Q[q:q + 1]), want[q:q + 1])


@pytest.mark.parametrize("threads,loads", [(256, 4), (384, 16), (512, 8)])
def test_self_join_takes_the_own_row_off(threads, loads, monkeypatch):
    import culsh_b200 as culsh
    monkeypatch.setenv("CULSH_CHAIN_BITS", "4096")
    monkeypatch.setenv("CULSH_CHAIN_THREADS", str(threads))
    monkeypatch.setenv("CULSH_CHAIN_LOADS", str(loads))
    rng = np.random.default_rng(2)
    n, d = 12_500, 6
    X = rng.standard_normal((n, d)).astype(np.float32)
    X[rng.permutation(n)[:1800]] = X[3]
    X[6000:8200] = X[3] + 10.0
    lsh = culsh.RPLSH(5, 9, seed=1)
    got, want = lsh.fit_query(X), lsh.fit(X).query(X)
    assert int(want.get_counts().max()) > 1800
    for f in ("get_offsets", "get_indices", "get_counts"):
        assert np.array_equal(getattr(got, f)(), getattr(want, f)())


@pytest.mark.parametrize("bounce", [1, 300_000, 5_000_000])
def test_result_inside_its_raw_array(bounce, monkeypatch):
    import culsh_b200 as culsh
    rng = np.random.default_rng(3)
    X = rng.standard_normal((200_000, 8)).astype(np.float32)
    Q = np.concatenate([rng.standard_normal((300, 8)), 1e3 * rng.standard_normal((30, 8)), X[:70]]).astype(np.float32)
    m = culsh.RPLSH(6, 5, seed=2).fit(X)  # about 37,000 entries a query: 60 MB raw
    want = m.query(Q)
    monkeypatch.setenv("CULSH_COMPACT_BOUNCE", str(bounce))
    got = m.query(Q)
    for f in ("get_offsets", "get_indices", "get_counts"):
        assert np.array_equal(getattr(got, f)(), getattr(want, f)())


def test_result_inside_its_raw_array_when_memory_is_short():
    """No memory for a second array of the result's size, and enough for the buffer."""
    import torch
    import culsh_b200 as culsh
    from culsh_b200 import _culsh_core as core_mod
    n, L, k, nq = 1_000_000, 4, 2, 200
    g = torch.Generator("cuda").manual_seed(4)
    X = torch.randn(n, 8, device="cuda", generator=g)
    Q = torch.randn(nq, 8, device="cuda", generator=g)
    core = core_mod.RPLSHCore(L, k, 2)
    m = culsh.RPLSH(L, k, seed=2).fit(X)
    want = m.query(Q)
    offsets, ids = want.get_offsets(), want.get_indices()
    stats = core.last_stats()
    raw, unique, launches = 4 * stats["raw_candidates"], 4 * stats["unique_candidates"], stats["launches"]
    assert unique > 400 << 20
    del want, X
    core.trim_scratch(0)
    torch.cuda.empty_cache()
    spare = raw + (200 << 20)
    ballast = torch.empty(torch.cuda.mem_get_info()[0] - spare, dtype=torch.uint8, device="cuda")
    try:
        got = m.query(Q)
        assert core.last_stats()["launches"] > launches
    finally:
        del ballast
        torch.cuda.empty_cache()
    assert np.array_equal(got.get_offsets(), offsets) and np.array_equal(got.get_indices(), ids)
    del got
    core.trim_scratch(0)


@pytest.mark.parametrize("threads", [256, 384, 512])
@pytest.mark.parametrize("L,n,bits", [(1, 20_000, 4096), (50, 20_000, 4096), (256, 9_000, 4096), (3, 300_000, 4096), (40, 300_000, None)])
def test_lists_cut_by_their_own_windows(L, n, bits, threads, monkeypatch):
    """Few sets: CTAs cut the lists themselves, more lists than they take at once, and more windows than sixty-four."""
    import culsh_b200 as culsh
    from culsh_b200 import _culsh_core as core_mod
    if bits:
        monkeypatch.setenv("CULSH_CHAIN_BITS", str(bits))
    monkeypatch.setenv("CULSH_CHAIN_THREADS", str(threads))
    rng = np.random.default_rng(L)
    d, k = 6, 5
    X = rng.standard_normal((n, d)).astype(np.float32)
    X[rng.permutation(n)[:1500]] = X[7]
    Q = np.concatenate([X[7:9], 1e3 * X[-1:]]).astype(np.float32)
    core = core_mod.RPLSHCore(L, k, 3)
    m = culsh.RPLSH(L, k, seed=3).fit(X)
    sig = lambda Y: core.hash(Y, m.index).transpose(1, 0, 2)  # noqa: E731
    want = _lists(m, sig(X), sig(Q), n, L)
    assert max(len(w) for w in want) >= 1500
    _assert_lists(m.query(Q), want)
    for q in range(len(Q)):
        _assert_lists(m.query(Q[q:q + 1]), want[q:q + 1])
