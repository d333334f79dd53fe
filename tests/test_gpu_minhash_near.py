"""Rows of 33 to 1,024 ids are hashed by a multiply-add each and settled by a few evaluations in full: lengths on both sides of
both lines and of whole eights, universes up to the bound and above it, ids beyond the stated universe, ids that repeat (their minima cannot be told
apart by the first form), one to eight hash functions a lane and more than one sweep, and rows next to shorter and to longer ones."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def _rows(lengths, d, rng, repeat=False):
    out = []
    for n in lengths:
        ids = rng.integers(0, d, n)
        if repeat:
            ids = ids[rng.integers(0, max(1, n // 5), n)]
        out.append(ids)
    return np.concatenate(out).astype(np.int32), np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)


def _check(core, indices, indptr, n, d, L, k):
    ix = core.fit(indices, indptr, n, d)
    sig = core.hash(indices, indptr, n, ix)
    want = oracle.minhash_signatures(indices, indptr, ix.get_hash_a(), ix.get_hash_b())
    assert np.array_equal(sig.transpose(1, 0, 2).reshape(n, L * k), want)


LENGTHS = [0, 1, 31, 32, 33, 34, 39, 40, 41, 64, 65, 110, 200, 255, 256, 257, 505, 511, 512, 513, 600, 1024, 1025, 1100, 1545]


@pytest.mark.parametrize("d", [3, 1 << 10, 50_000, 1 << 16, 1 << 20, (1 << 20) + 1, 1 << 22, 1 << 23, (1 << 31) - 1])
@pytest.mark.parametrize("repeat", [False, True])
def test_lengths_and_universes(d, repeat):
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(d % 97)
    lengths = rng.permutation(LENGTHS * 12)
    indices, indptr = _rows(lengths, d, rng, repeat)
    _check(core_mod.MinHashCore(16, 4, 5), indices, indptr, len(lengths), d, 16, 4)


@pytest.mark.parametrize("L,k", [(1, 3), (8, 4), (8, 8), (10, 9), (16, 8), (20, 8), (24, 8), (28, 8), (32, 8), (40, 10)])
def test_functions_of_a_lane(L, k):
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(L)
    lengths = rng.integers(20, 200, 300)
    indices, indptr = _rows(lengths, 1 << 20, rng)
    _check(core_mod.MinHashCore(L, k, 9), indices, indptr, 300, 1 << 20, L, k)


def test_ids_beyond_the_stated_universe():
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(3)
    lengths = rng.integers(30, 120, 400)
    lengths[::9] = rng.integers(500, 1200, len(lengths[::9]))  # far ids in the first list of a row or in a later one
    indices, indptr = _rows(lengths, 1 << 16, rng)
    far = rng.random(len(indices)) < 0.002
    indices[far] = rng.integers(1 << 16, 1 << 30, int(far.sum()))
    _check(core_mod.MinHashCore(8, 4, 1), indices, indptr, 400, 1 << 16, 8, 4)


def test_many_rows():
    """Enough minima for those that are evaluated again to be among them in number."""
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(4)
    lengths = rng.integers(33, 300, 6000)
    indices, indptr = _rows(lengths, 1 << 22, rng)
    _check(core_mod.MinHashCore(32, 4, 2), indices, indptr, 6000, 1 << 22, 32, 4)


def _around_the_last_id(a, b, m, alike, rng):
    """A row that ends with `m` ids whose mean is its last id and whose first forms are within 2^18 of each other, while that of the last id is far
    from them.  With the last eight filled up by copies of the last id there are as many of it as of the ids around it, and their sums are the
    same.  The values of all other ids are above those of both."""
    p, alpha = oracle.MINHASH_PRIME, (int(a) * 2 ** 32 + oracle.MINHASH_PRIME // 2) // oracle.MINHASH_PRIME
    f = lambda c: (int(a) * c + int(b)) % p  # noqa: E731
    D = np.arange(1, 1 << 19, dtype=np.uint64)
    y = D * np.uint64(alpha) & np.uint64(0xFFFFFFFF)
    off = y * np.uint64(m) & np.uint64(0xFFFFFFFF)
    off = np.minimum(off, np.uint64(2 ** 32) - off)
    off[(y < 2 ** 28) | (y > 2 ** 32 - 2 ** 28)] = 2 ** 32
    D = int(D[np.argmin(off)])
    if off.min() >= 2 ** 18:
        return None  # no such distance for this function
    while True:
        last = int(rng.integers(1 << 19, 1 << 20))
        near = [last - D] * (m - 1) + [last + (m - 1) * D]
        if f(near[0]) < 2 ** 30 and f(near[0]) + 2 ** 24 < f(last) < 0.95 * p:
            break
    others = []
    while len(others) < 40 - 2 * m:  # 32, and those that leave room in the last eight for m, one and m - 1
        c = int(rng.integers(0, 1 << 21))
        if f(c) > f(last) + 2 ** 24:
            others.append(c)
    row = others[:1] * len(others) if alike else others
    assert min(map(f, row + near + [last])) in map(f, near) and (len(row) + m + 1) % 8 == 9 - m
    return row + near + [last]


@pytest.mark.parametrize("alike", [False, True])
@pytest.mark.parametrize("m", [2, 3, 4])
def test_ids_around_the_last_one(m, alike):
    """For each hash function a row whose least ones have the last id, which stands for the places behind it, in their middle."""
    from culsh_b200 import _culsh_core as core_mod
    L, k, d = 8, 4, 1 << 22
    rng = np.random.default_rng(m)
    for seed in (0, 42):
        core = core_mod.MinHashCore(L, k, seed)
        ix = core.fit(np.arange(40, dtype=np.int32), np.array([0, 40], np.int32), 1, d)
        rows = [_around_the_last_id(a, b, m, alike, rng) for a, b in zip(ix.get_hash_a().ravel(), ix.get_hash_b().ravel())]
        rows = [r for r in rows if r]
        assert len(rows) > 3 * L * k // 4
        indices = np.concatenate(rows).astype(np.int32)
        indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
        _check(core, indices, indptr, len(rows), d, L, k)


@pytest.mark.parametrize("alike", [0, 1, 3, 8, 31, 1000])
@pytest.mark.parametrize("late", [False, True])
def test_rows_that_repeat_ids(alike, late):
    """On both sides of the line from which rows that repeat ids, and those behind them, are done in the other forms, with the repeated ones among a row's first
    32 or behind them, next to rows that do not."""
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(alike)
    rows = []
    for n in [33, 34, 64, 65, 200, 1024] * 20:
        ids = rng.permutation(1 << 20)[:n]
        first = 32 if late else 0
        for j in range(min(alike, n - first - 1)):
            ids[first + 1 + j] = ids[rng.integers(0, first + 1 + j)]
        rows += [ids, rng.permutation(1 << 20)[:int(rng.integers(20, 80))]]
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    _check(core_mod.MinHashCore(16, 8, 3), np.concatenate(rows).astype(np.int32), indptr, len(rows), 1 << 20, 16, 8)
