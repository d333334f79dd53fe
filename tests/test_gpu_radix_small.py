"""One CTA sorts a table of up to 12,288 rows (8,192 with a two-word key that is not compressed): row counts
at the edges of a warp, of the 1024-item step and of those lines, all key widths, against a sort on the host.
The collections repeat rows, so that equal keys show whether rows keep their order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 33, 1023, 1024, 1025, 8191, 8192, 8193, 12_287, 12_288, 12_289]


def _check(ix, sig, n, L):
    cand, tab = ix.get_candidate_indices(), ix.get_table_bucket_offsets()
    off, keys = ix.get_bucket_candidate_offsets(), ix.get_bucket_signatures().reshape(ix.n_total_buckets, -1)
    for t in range(L):
        raw = np.ascontiguousarray(sig[t]).view(np.uint8).reshape(n, -1)
        order = np.lexsort(tuple(raw[:, j] for j in range(raw.shape[1] - 1, -1, -1)))
        assert np.array_equal(cand[t * n:(t + 1) * n], order)
        srt = raw[order]
        head = np.concatenate([[True], (srt[1:] != srt[:-1]).any(axis=1)])
        assert np.array_equal(keys[tab[t]:tab[t + 1]], srt[head])
        assert np.array_equal(off[tab[t]:tab[t + 1]], t * n + np.flatnonzero(head))


def _rows(n, scale):
    rng = np.random.default_rng(n)
    base = scale * rng.standard_normal((max(1, n // 3), 12))
    return base[rng.integers(0, len(base), n)].astype(np.float32)


@pytest.mark.parametrize("k", [5, 24, 40, 100])
@pytest.mark.parametrize("n", SIZES)
def test_sign_keys(n, k):
    from culsh_b200 import _culsh_core as core_mod
    X = _rows(n, 1.0)
    core = core_mod.RPLSHCore(3, k, 4)
    ix = core.fit_float(X, n, 12)
    _check(ix, core.hash(X, ix), n, 3)


@pytest.mark.parametrize("k,scale", [(3, 1.0), (8, 1.0), (8, 9.0), (11, 1.0), (8, 60.0)])
@pytest.mark.parametrize("n", SIZES)
def test_p_stable_keys(n, k, scale):
    from culsh_b200 import _culsh_core as core_mod
    X = _rows(n, scale)
    core = core_mod.PSLSHCore(3, k, 2, 4)
    ix = core.fit_float(X, n, 12)
    _check(ix, core.hash(X, ix), n, 3)


@pytest.mark.parametrize("k", [1, 2, 3, 16])
@pytest.mark.parametrize("n", SIZES)
def test_minhash_keys(n, k):
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(n)
    indices = rng.integers(0, 60, 3 * n).astype(np.int32)
    indptr = (3 * np.arange(n + 1)).astype(np.int32)
    core = core_mod.MinHashCore(3, k, 4)
    ix = core.fit(indices, indptr, n, 60)
    _check(ix, core.hash(indices, indptr, n, ix), n, 3)


@pytest.mark.parametrize("family,k,scale", [("rp", 40, 1.0), ("rp", 100, 1.0), ("ps", 8, 1.0), ("ps", 8, 9.0), ("ps", 8, 60.0), ("ps", 11, 1.0), ("mh", 2, 0), ("mh", 3, 0),
                                            ("mh", 16, 0)])
@pytest.mark.parametrize("n", [n for n in SIZES if n <= 8192])
def test_without_splitters(n, family, k, scale, monkeypatch):
    """Keys of two words and more in up to 2,048 rows are sorted by splitters as a rule, and longer tables by clusters of CTAs where they are
    few: with a CTA for each as before.  (The rows and hashes of the tests above: wider spreads make values on which `hash`, which computes all of them
    in full width, and the fit differ by their rounding.)"""
    from culsh_b200 import _culsh_core as core_mod
    monkeypatch.setenv("CULSH_SORT_SPLITTERS", "0")
    L = 3 if n < 2048 else 33
    cores = {"rp": lambda: core_mod.RPLSHCore(L, k, 4), "ps": lambda: core_mod.PSLSHCore(L, k, 2, 4), "mh": lambda: core_mod.MinHashCore(L, k, 4)}
    core = cores[family]()
    if family == "mh":
        rng = np.random.default_rng(n)
        indices = rng.integers(0, 60, 3 * n).astype(np.int32)
        indptr = (3 * np.arange(n + 1)).astype(np.int32)
        ix = core.fit(indices, indptr, n, 60)
        stats, sig = core.last_stats(), core.hash(indices, indptr, n, ix)
    else:
        X = _rows(n, scale)
        ix = core.fit_float(X, n, 12)
        stats, sig = core.last_stats(), core.hash(X, ix)
    assert stats["sort_ctas"] == 1
    _check(ix, sig, n, 3)
