"""Keys of four words and more are sorted word by word, tables of more than 12,288 rows and, with the one-CTA sort
switched off, shorter ones: row counts on both sides of the 4096-item tile, of the 96 tiles from which tile offsets
are scanned in chunks, and of whole chunks of 64 tiles, key lengths that end inside a word (16 to 64
bytes, 8-word keys among them), and collections where the rows agree in the leading, the trailing or all hashes, so that
the order depends on every word and equal keys keep their row order.  The chunked scan of one- and
two-word keys (tiles of 4096 and 3072) is checked at the same counts of tiles."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


TILE = 4096


@pytest.mark.parametrize("n,k", [(1, 3), (31, 16), (4095, 3), (4096, 4), (4097, 5), (8193, 8), (12_289, 9), (12_289, 5), (20_000, 16),
                                 (20_000, 8), (95 * TILE, 5), (95 * TILE + 1, 3), (96 * TILE + 1, 8), (128 * TILE, 3),
                                 (128 * TILE + 1, 4), (2_097_153, 3)])
def test_index_equals_oracle_order(n, k, monkeypatch):
    from culsh_b200 import _culsh_core as core_mod
    if n <= 12_288:
        monkeypatch.setenv("CULSH_SORT_NO_PACK", "1")
    rng = np.random.default_rng(n)
    L = 2
    # row r of block b has b's set of ids with a few of the positions changed: many equal hashes
    sets = rng.integers(0, 400, (max(1, n // 50), 6))
    rows = sets[rng.integers(0, len(sets), n)]
    hit = rng.random(n) < 0.3
    rows[hit, rng.integers(0, 6, int(hit.sum()))] = rng.integers(0, 400, int(hit.sum()))
    indices = np.ascontiguousarray(rows.astype(np.int32)).ravel()
    indptr = (6 * np.arange(n + 1)).astype(np.int32)
    core = core_mod.MinHashCore(L, k, 7)
    ix = core.fit(indices, indptr, n, 400)
    sig = core.hash(indices, indptr, n, ix)  # [L][n][k]
    # the order of the engine: unsigned bytes in memory order, ties by row
    got_c, got_b = ix.get_candidate_indices(), ix.get_bucket_signatures().reshape(-1, 4 * k)
    off, tab = ix.get_bucket_candidate_offsets(), ix.get_table_bucket_offsets()
    for t in range(L):
        raw = np.ascontiguousarray(sig[t]).view(np.uint8).reshape(n, 4 * k)
        big = np.ascontiguousarray(raw).view(">u4")
        order = np.lexsort(tuple(big[:, j] for j in range(k - 1, -1, -1)))
        assert np.array_equal(got_c[t * n:(t + 1) * n], order)
        srt = raw[order]
        head = np.concatenate([[True], (srt[1:] != srt[:-1]).any(axis=1)])
        assert np.array_equal(got_b[tab[t]:tab[t + 1]], srt[head])
        assert np.array_equal(off[tab[t]:tab[t + 1]], t * n + np.flatnonzero(head))
    want = oracle.minhash_signatures(indices[:600], indptr[:min(n, 100) + 1], ix.get_hash_a(), ix.get_hash_b())
    assert np.array_equal(sig[:, :min(n, 100)].transpose(1, 0, 2).reshape(-1, L * k), want)


@pytest.mark.parametrize("k,tile", [(16, 4096), (40, 3072)])
@pytest.mark.parametrize("tiles,extra", [(95, 0), (95, 1), (96, 0), (96, 1), (128, 0), (128, 1), (192, -1)])
def test_scan_of_many_tiles(k, tile, tiles, extra):
    """Sign keys of one and two words: the index against a stable sort of the signatures on the host."""
    from culsh_b200 import _culsh_core as core_mod
    n, d, L = tiles * tile + extra, 8, 2
    rng = np.random.default_rng(n)
    base = rng.standard_normal((n // 3 + 1, d)).astype(np.float32)  # every row about three times
    X = base[rng.integers(0, len(base), n)]
    core = core_mod.RPLSHCore(L, k, 5)
    ix = core.fit_float(X, n, d)
    sig = core.hash(X, ix)  # [L][n][k] bytes
    cand = ix.get_candidate_indices()
    for t in range(L):
        key = (sig[t].astype(np.uint64) << np.arange(k - 1, -1, -1, dtype=np.uint64)).sum(axis=1, dtype=np.uint64)
        assert np.array_equal(cand[t * n:(t + 1) * n], np.argsort(key, kind="stable"))


@pytest.mark.parametrize("n,k", [(1, 3), (31, 16), (4095, 3), (4096, 4), (4097, 5), (8193, 8), (12_289, 9), (12_289, 5), (20_000, 16),
                                 (20_000, 8), (95 * TILE, 5), (95 * TILE + 1, 3), (96 * TILE + 1, 8), (128 * TILE, 3),
                                 (128 * TILE + 1, 4), (2_097_153, 3)])
def test_word_by_word(n, k, monkeypatch):
    """As above with splitters, which take keys of two words and more in up to four million rows as a rule, and the sorts in one launch switched off."""
    from culsh_b200 import _culsh_core as core_mod
    monkeypatch.setenv("CULSH_SORT_SPLITTERS", "0")
    monkeypatch.setenv("CULSH_SORT_NO_PACK", "1")
    stats = []

    class Core(core_mod.MinHashCore):
        def fit(self, *args, **kw):
            ix = super().fit(*args, **kw)
            stats.append(self.last_stats())
            return ix
    monkeypatch.setattr(core_mod, "MinHashCore", Core)
    test_index_equals_oracle_order(n, k, monkeypatch)
    assert len(stats) == 1 and stats[0]["sort_ctas"] == 0 and stats[0]["sort_passes"] == 4 * k
