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
