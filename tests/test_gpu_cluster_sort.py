"""Short tables are sorted by a cluster of CTAs each, eight or four of them by the number of tables: row counts that
leave the last CTA full, with one row, or empty, the fewest a cluster takes and the most its CTAs hold, for each
form of the keys, against a stable sort on the host.  Rows come about three times, so that equal keys show whether rows keep
their order; a third of the hashes is the same for all rows, so that a digit has all items of a warp."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(ix, sig, n, L):
    cand = ix.get_candidate_indices()
    for t in range(L):
        raw = np.ascontiguousarray(sig[t]).view(np.uint8).reshape(n, -1)
        order = np.lexsort(tuple(raw[:, j] for j in range(raw.shape[1] - 1, -1, -1)))
        assert np.array_equal(cand[t * n:(t + 1) * n], order)


SHAPES = [(1, 2), (1000, 8), (2047, 13), (2048, 13), (2049, 16), (4095, 13), (4096, 13), (4097, 13), (4353, 5), (8191, 32), (8192, 32),
          (8193, 16), (12_288, 33), (12_289, 33), (24_576, 16), (24_577, 16), (16_384, 14), (16_385, 14), (32_768, 4), (32_769, 4),
          (49_152, 13), (49_153, 13), (10_000, 150)]


@pytest.mark.parametrize("n,L", SHAPES)
@pytest.mark.parametrize("family,k,scale", [("rp", 13, 1.0), ("rp", 40, 1.0), ("ps", 8, 1.0), ("ps", 3, 1.0), ("ps", 8, 30.0)])
def test_order_of_the_host(n, L, family, k, scale):
    from culsh_b200 import _culsh_core as core_mod
    d = 8
    rng = np.random.default_rng(n + k)
    base = (scale * rng.standard_normal((n // 3 + 1, d))).astype(np.float32)
    X = base[rng.integers(0, len(base), n)]
    X[:, 0] = 40.0 * scale if family == "rp" else 0.0
    core = core_mod.RPLSHCore(L, k, 5) if family == "rp" else core_mod.PSLSHCore(L, k, 2, 5)
    ix = core.fit_float(X, n, d)
    _check(ix, core.hash(X, ix), n, L)


@pytest.mark.parametrize("n,L", SHAPES)
@pytest.mark.parametrize("k", [3, 5, 9])
def test_wide_keys(n, L, k):
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(n + k)
    sets = rng.integers(0, 400, (n // 3 + 1, 6)).astype(np.int32)
    indices = np.ascontiguousarray(sets[rng.integers(0, len(sets), n)]).ravel()
    indptr = (6 * np.arange(n + 1)).astype(np.int32)
    core = core_mod.MinHashCore(L, k, 7)
    ix = core.fit(indices, indptr, n, 400)
    _check(ix, core.hash(indices, indptr, n, ix), n, L)


@pytest.mark.parametrize("n,L", SHAPES)
@pytest.mark.parametrize("k", [3, 5, 9])
def test_wide_keys_without_splitters(n, L, k, monkeypatch):
    """Splitters take wide keys of up to 2,048 and from 12,289 or 16,385 rows on as a rule."""
    from culsh_b200 import _culsh_core as core_mod
    monkeypatch.setenv("CULSH_SORT_SPLITTERS", "0")
    stats = []

    class Core(core_mod.MinHashCore):
        def fit(self, *args, **kw):
            ix = super().fit(*args, **kw)
            stats.append(self.last_stats())
            return ix
    monkeypatch.setattr(core_mod, "MinHashCore", Core)
    test_wide_keys(n, L, k)
    ctas = 8 if L <= 13 and 4096 <= n <= 49_152 else 4 if L <= 32 and 8192 <= n <= 24_576 else int(n <= 12_288 and L <= 148)
    assert [s["sort_ctas"] for s in stats] == [ctas]


@pytest.mark.parametrize("n,L,ctas", [(1000, 8, 1), (10_000, 13, 8), (24_576, 32, 4), (49_152, 13, 8), (49_153, 13, 0)])
def test_stats_name_the_form(n, L, ctas):
    from culsh_b200 import _culsh_core as core_mod
    core = core_mod.RPLSHCore(L, 12, 1)
    core.fit_float(np.random.default_rng(n).standard_normal((n, 8)).astype(np.float32), n, 8)
    assert core.last_stats()["sort_ctas"] == ctas
