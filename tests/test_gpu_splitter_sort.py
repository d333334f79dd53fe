"""Keys of two words and more are sorted by sampled splitters, word by word by radix passes or, as one bin, by one CTA: row
counts on both sides of a bin, of the change from one to several chunks of samples and of a tile, keys that end inside
their words, and collections in which all rows are alike, come in order, repeat with a period or differ in one hash only, so that bins
are full of equal keys and some are sorted in pieces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(core, ix, indices, indptr, n, L, k):
    sig = core.hash(indices, indptr, n, ix)  # [L][n][k]
    got, keys = ix.get_candidate_indices(), ix.get_bucket_signatures().reshape(-1, 4 * k)
    off, tab = ix.get_bucket_candidate_offsets(), ix.get_table_bucket_offsets()
    for t in range(L):
        raw = np.ascontiguousarray(sig[t]).view(np.uint8).reshape(n, 4 * k)
        big = raw.view(">u4")
        order = np.lexsort(tuple(big[:, j] for j in range(k - 1, -1, -1)))
        assert np.array_equal(got[t * n:(t + 1) * n], order)
        srt = raw[order]
        head = np.concatenate([[True], (srt[1:] != srt[:-1]).any(axis=1)])
        assert np.array_equal(keys[tab[t]:tab[t + 1]], srt[head])
        assert np.array_equal(off[tab[t]:tab[t + 1]], t * n + np.flatnonzero(head))


def _rows(kind, n, rng):
    if kind == "alike":
        return np.tile(rng.integers(0, 400, 6), (n, 1))
    if kind == "few":  # two sets, one of them rare
        return rng.integers(0, 400, (2, 6))[(rng.random(n) < 0.01).astype(int)]
    if kind == "period":
        return rng.integers(0, 4000, (7, 6))[np.arange(n) % 7]
    if kind == "last":  # every row starts with the same ids
        return np.concatenate([np.tile(rng.integers(0, 50, 5), (n, 1)), rng.integers(0, 1 << 19, (n, 1))], axis=1)
    if kind == "near":  # sets of 30 ids that differ in one: most hashes are the same in all rows
        return np.concatenate([np.tile(np.arange(29), (n, 1)), rng.integers(0, max(2, n // 8), (n, 1))], axis=1)
    if kind == "but one":  # in the last place, in the first or in the middle
        rows = np.tile(rng.integers(0, 400, 6), (n, 1))
        rows[rng.choice([0, n // 2, n - 1])] += 1
        return rows
    rows = rng.integers(0, 1 << 19, (max(1, n // 40), 6))[rng.integers(0, max(1, n // 40), n)]
    if kind == "sorted":
        return rows[np.lexsort(rows.T)]
    change = rng.random(n) < 0.4
    rows[change, rng.integers(0, 6, int(change.sum()))] = rng.integers(0, 1 << 19, int(change.sum()))
    return rows


@pytest.mark.parametrize("splitters", [None, "1", "0"])
@pytest.mark.parametrize("n,k,kind", [
    (1, 3, "mixed"), (9, 4, "mixed"), (2047, 4, "mixed"), (2048, 16, "mixed"), (2048, 4, "alike"), (2049, 4, "mixed"), (3000, 9, "few"),
    (16_384, 4, "mixed"), (16_385, 5, "period"), (20_000, 4, "alike"), (20_000, 4, "sorted"), (65_537, 3, "last"),
    (1500, 2, "mixed"), (12_289, 2, "few"), (100_003, 2, "sorted"), (700_000, 2, "mixed"), (100_003, 8, "mixed"), (100_003, 4, "few"), (524_288, 4, "mixed"), (524_289, 4, "sorted"), (600_000, 6, "last"), (2_100_000, 3, "mixed")])
def test_order(n, k, kind, splitters, monkeypatch):
    from culsh_b200 import _culsh_core as core_mod
    if splitters:
        monkeypatch.setenv("CULSH_SORT_SPLITTERS", splitters)
    rng = np.random.default_rng(n + k)
    L = 2
    indices = np.ascontiguousarray(_rows(kind, n, rng).astype(np.int32)).ravel()
    indptr = (6 * np.arange(n + 1)).astype(np.int32)
    core = core_mod.MinHashCore(L, k, 7)
    _check(core, core.fit(indices, indptr, n, 1 << 19), indices, indptr, n, L, k)


@pytest.mark.parametrize("n,k,kind", [
    (300, 5, "alike"), (300, 16, "but one"), (2048, 8, "alike"), (2048, 5, "near"), (2047, 9, "near"), (2048, 16, "but one"), (5000, 16, "alike"), (20_000, 5, "near"),
    (20_000, 16, "near"), (20_000, 8, "alike"), (40_000, 7, "few"), (40_000, 12, "but one"), (300_000, 5, "few"), (300_000, 8, "near"), (300_000, 10, "period")])
def test_wide_keys_that_repeat(n, k, kind, monkeypatch):
    """Keys of eight and sixteen words whose first words are the same in all rows of a bin or in many: the words behind them are looked at only
    where there are rows that are not alike."""
    from culsh_b200 import _culsh_core as core_mod
    monkeypatch.setenv("CULSH_SORT_SPLITTERS", "1")
    rng = np.random.default_rng(n + k)
    rows = _rows(kind, n, rng)
    indices = np.ascontiguousarray(rows.astype(np.int32)).ravel()
    indptr = (rows.shape[1] * np.arange(n + 1)).astype(np.int32)
    core = core_mod.MinHashCore(2, k, 7)
    _check(core, core.fit(indices, indptr, n, 1 << 19), indices, indptr, n, 2, k)


def _largest_bin(order, n):
    """Rows of the fullest bin of a table whose rows come in this order, from the rows that the sort takes as samples."""
    bins = 1
    while bins * 1024 < n:
        bins *= 2
    samples = max(512, 8 * bins)
    g = np.arange(samples, dtype=np.uint64)
    r0, r1 = g * np.uint64(n) // np.uint64(samples), (g + np.uint64(1)) * np.uint64(n) // np.uint64(samples)
    h = (g.astype(np.uint32) + np.uint32(1)) * np.uint32(0x9E3779B9)
    for shift, factor in ((16, 0x85EBCA6B), (13, 0xC2B2AE35), (16, 1)):
        h = (h ^ (h >> np.uint32(shift))) * np.uint32(factor)
    place = np.empty(n, np.int64)
    place[order] = np.arange(n)
    at = np.sort(place[(r0 + h % (r1 - r0)).astype(np.int64)])[samples // bins::samples // bins]
    return int(np.diff(np.concatenate([[0], at, [n]])).max())


@pytest.mark.parametrize("n,k,kind", [(524_288, 2, "mixed"), (1_048_576, 2, "mixed"), (524_288, 3, "last"), (524_288, 6, "mixed"), (524_288, 8, "near"), (524_288, 9, "last"), (524_288, 16, "near")])
def test_bins_in_pieces(n, k, kind, monkeypatch):
    """Tables whose bins hold 1,024 rows on average, so that some hold more than the 2,048 that a CTA sorts at once.  (Not where
    few keys differ: rows that are alike come in the order of their ids, which the samples cover evenly.)"""
    from culsh_b200 import _culsh_core as core_mod
    monkeypatch.setenv("CULSH_SORT_SPLITTERS", "1")  # two long tables of short keys are not theirs as a rule
    rng = np.random.default_rng(k)
    rows = _rows(kind, n, rng)
    indices = np.ascontiguousarray(rows.astype(np.int32)).ravel()
    indptr = (rows.shape[1] * np.arange(n + 1)).astype(np.int32)
    core = core_mod.MinHashCore(2, k, 7)
    ix = core.fit(indices, indptr, n, 1 << 19)
    assert core.last_stats()["sort_ctas"] == -1
    _check(core, ix, indices, indptr, n, 2, k)
    order = ix.get_candidate_indices()  # as _check has found it to be
    assert max(_largest_bin(order[t * n:(t + 1) * n], n) for t in range(2)) > 2048


@pytest.mark.parametrize("n,k,L,route", [(16_384, 3, 32, 4), (16_385, 3, 32, -1), (12_288, 4, 32, 4), (12_289, 4, 32, -1), (12_289, 8, 32, -1), (2048, 3, 32, -1), (2049, 3, 32, 1),
                                         (524_288, 2, 7, -1), (524_289, 2, 7, 0), (2_097_152, 2, 8, -1), (2_097_153, 2, 8, 0), (2_097_153, 3, 1, -1)])
def test_which_sort(n, k, L, route):
    """Lines between the sorts: clusters of four CTAs, one CTA, passes with launches of their own and splitters."""
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(n)
    indices, indptr = rng.integers(0, 1 << 19, 6 * n).astype(np.int32), (6 * np.arange(n + 1)).astype(np.int32)
    core = core_mod.MinHashCore(L, k, 7)
    core.fit(indices, indptr, n, 1 << 19)
    assert core.last_stats()["sort_ctas"] == route


def test_wide_p_stable_keys_and_many_tables():
    """Values of two bytes (keys of four words with zeros in front), in more tables than the chip has SMs, and of one byte that span too much for the
    compressed sort."""
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(1)
    for n, L, k, scale in [(3000, 150, 5, 300), (50_000, 2, 12, 300), (1500, 3, 8, 6), (12_288, 40, 8, 6), (100_003, 2, 7, 6)]:
        X = (scale * rng.standard_normal((n, 6))).astype(np.float32)
        core = core_mod.PSLSHCore(L, k, 1, 3)
        ix = core.fit_float(X, n, 6)
        assert ix.elem_bytes == (2 if scale == 300 else 1)
        sig, got = core.hash(X, ix), ix.get_candidate_indices()
        for t in range(0, L, 37):
            raw = np.ascontiguousarray(sig[t]).view(np.uint8).reshape(n, 4 * k)
            order = np.lexsort(tuple(raw[:, j] for j in range(4 * k - 1, -1, -1)))
            assert np.array_equal(got[t * n:(t + 1) * n], order)

@pytest.mark.parametrize("n,k,L,route", [(114_688, 7, 8, -1), (114_689, 7, 8, 0), (49_152, 9, 8, 8), (49_153, 9, 8, -1), (32_768, 10, 8, 8), (32_769, 10, 8, -1), (32_769, 11, 8, -1),
                                         (1_048_576, 9, 7, -1), (1_048_577, 9, 7, 0), (1_048_577, 9, 8, -1), (2_097_152, 10, 4, -1), (2_097_153, 10, 4, 0), (2_097_153, 11, 3, 0), (2_097_153, 11, 4, -1)])
def test_which_sort_of_one_byte_values(n, k, L, route):
    """As above, for keys of as many bytes as hashes, whose values span too much for the compressed form."""
    import torch
    from culsh_b200 import _culsh_core as core_mod
    X = 9 * torch.randn(n, 4, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    torch.cuda.synchronize()
    core = core_mod.PSLSHCore(L, k, 2, 3)
    assert core.fit_float(X, n, 4).elem_bytes == 1
    assert core.last_stats()["sort_ctas"] == route



def test_no_scratch_where_another_sort_runs():
    """Four million keys of eight bytes that are sorted in compressed form: the handle holds no more for them than for one row more, which the splitters do not
    take in any form."""
    import torch
    from culsh_b200 import _culsh_core as core_mod
    held = []
    X = torch.randn(4_194_305, 4, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    core = core_mod.PSLSHCore(16, 8, 2, 3)
    for n in (4_194_304, 4_194_305):
        core.trim_scratch(0)
        ix = core.fit_float(X[:n], n, 4)
        assert core.last_stats()["sort_ctas"] == 0 and core.last_stats()["sort_passes"] == 5
        del ix
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        core.trim_scratch(0)
        held.append(torch.cuda.mem_get_info()[0] - free)
    assert held[0] <= held[1], held
