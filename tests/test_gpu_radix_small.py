"""One CTA sorts a table of up to 12,288 rows (8,192 with a two-word key that is not compressed): row counts
at the edges of a warp, of the 1024-item step and of those lines, all key widths, against a sort on the host.
The collections repeat rows, so that equal keys show whether rows keep their order.  Once as they come - keys of two words and more in up to 2,048
rows are sorted by splitters then - and once without splitters."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 33, 1023, 1024, 1025, 8191, 8192, 8193, 12_287, 12_288, 12_289]


@pytest.fixture(params=[None, "0"], autouse=True)
def splitters(request, monkeypatch):
    if request.param:
        monkeypatch.setenv("CULSH_SORT_SPLITTERS", request.param)
    return request.param


def _tables(n):
    """From 2,048 rows on as many as leave a CTA for each: fewer are sorted by clusters."""
    return 3 if n < 2048 else 33


def _check(core, ix, sig, n, L, splitters):
    if splitters and n <= 8192:
        assert core.last_stats()["sort_ctas"] == 1
    cand, tab = ix.get_candidate_indices(), ix.get_table_bucket_offsets()
    off, keys = ix.get_bucket_candidate_offsets(), ix.get_bucket_signatures().reshape(ix.n_total_buckets, -1)
    for t in range(0, L, 1 if L < 8 else 16):
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
def test_sign_keys(n, k, splitters):
    from culsh_b200 import _culsh_core as core_mod
    X = _rows(n, 1.0)
    core = core_mod.RPLSHCore(_tables(n), k, 4)
    ix = core.fit_float(X, n, 12)
    sig = core.hash(X, ix)
    _check(core, ix, sig, n, _tables(n), splitters)


@pytest.mark.parametrize("k,scale", [(3, 1.0), (8, 1.0), (8, 9.0), (11, 1.0), (8, 60.0)])
@pytest.mark.parametrize("n", SIZES)
def test_p_stable_keys(n, k, scale, splitters):
    from culsh_b200 import _culsh_core as core_mod
    X = _rows(n, scale)
    core = core_mod.PSLSHCore(_tables(n), k, 2, 4)
    ix = core.fit_float(X, n, 12)
    sig = core.hash(X, ix)
    _check(core, ix, sig, n, _tables(n), splitters)


@pytest.mark.parametrize("k", [1, 2, 3, 16])
@pytest.mark.parametrize("n", SIZES)
def test_minhash_keys(n, k, splitters):
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(n)
    indices = rng.integers(0, 60, 3 * n).astype(np.int32)
    indptr = (3 * np.arange(n + 1)).astype(np.int32)
    core = core_mod.MinHashCore(_tables(n), k, 4)
    ix = core.fit(indices, indptr, n, 60)
    sig = core.hash(indices, indptr, n, ix)
    _check(core, ix, sig, n, _tables(n), splitters)
