"""Lookups go through keys of the table that are laid out in shared memory (256 of one word, 128 of two, ... 16 of
sixteen) and search on from the nearest one.  Numbers of buckets
on both sides of those counts and of their multiples, queries below, between, at and above the keys of a table, more queries
than a CTA has threads, against a search on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 3, 6, 13])  # MinHash keys of 1, 2, 4, 8 and 16 words
@pytest.mark.parametrize("values", [1, 15, 16, 17, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 513, 3000])
def test_against_the_host(k, values):
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(values)
    L, copies = 9, 1 + 40 // values
    n = values * copies
    ids = np.repeat(rng.permutation(1 << 20)[:2 * values:2], copies)[rng.permutation(n)].astype(np.int32)
    core = core_mod.MinHashCore(L, k, 3)
    ix = core.fit(ids, np.arange(n + 1, dtype=np.int32), n, 1 << 20)
    nq = 1000  # 9,000 pairs: beyond what is looked up and counted in one launch
    q = np.concatenate([rng.choice(ids, 500), rng.integers(0, 1 << 20, 500)]).astype(np.int32)
    got = core.query(q, np.arange(nq + 1, dtype=np.int32), nq, ix)
    sx, sq = core.hash(ids, np.arange(n + 1, dtype=np.int32), n, ix), core.hash(q, np.arange(nq + 1, dtype=np.int32), nq, ix)
    off, cand = got.get_offsets().astype(np.int64), got.get_indices()
    for i in range(nq):
        hit = (sx == sq[:, i:i + 1]).all(axis=2).any(axis=0)
        assert np.array_equal(cand[off[i]:off[i + 1]], np.flatnonzero(hit))
