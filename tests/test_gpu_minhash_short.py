"""MinHash rows of at most 1024 ids hash ids below 2^16 without the wrap of the fold and evaluate a minimum below
5 * (2^16 + 1) again: parameters that put single ids at the prime, at zero and on both sides of that line, with and without a
wrap, ids on both sides of 2^16 and of 2^20 alone and mixed inside one 32-id step, rows on both sides of 1024 ids, numbers of hash
functions that leave lanes without one, against the 64-bit oracle."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,k", [(4, 1), (3, 11), (8, 8), (16, 8), (9, 9), (32, 8), (36, 8)])
def test_minima_around_the_line(L, k):
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(L * k)
    line, top = 1 << 16, 1 << 22
    again = 5 * (line + 1)
    ids = [0, 1, 7, line - 2, line - 1, line, line + 1, (1 << 20) - 1]
    rows = [[c] for c in ids] + [[], ids, ids[:-1], ids + [1 << 20], list(range(line - 20, line + 12)), list(range(line - 33, line))]
    rows += [sorted(rng.choice(line, n, replace=False)) for n in (31, 33, 64, 1023, 1024, 1025, 3000)]
    rows += [sorted(rng.choice(1 << 20, n, replace=False)) for n in (31, 200, 1024, 1025)]
    rows += [list(rng.permutation(np.concatenate([rng.choice(line, 40, replace=False), line + rng.choice(line, 40, replace=False)])))]
    H, p = L * k, oracle.MINHASH_PRIME
    A = rng.integers(1, p, H).astype(np.uint32)
    B = rng.integers(0, p, H).astype(np.uint32)
    A[H - 1] = B[H - 1] = p - 1
    values = [0, 1, 4, 5, p - 1, p - 5, p - 6, again - 6, again - 5, again - 4, again, again + 1, line, 1000]
    for h in range(H - 1):
        c, v = ids[h % len(ids)], values[(h // 2) % len(values)]
        if h % 3:
            B[h] = (v - int(A[h]) * c) % p
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    indices = np.array([c for r in rows for c in r], dtype=np.int32)
    want = oracle.minhash_signatures(indices, indptr, A, B)
    oidx = oracle.fit_index(want, L, k)
    ix = core_mod.MinHashIndex.load(
        candidate_indices=oidx.candidate_indices, bucket_signatures=oidx.bucket_signatures,
        bucket_candidate_offsets=oidx.bucket_candidate_offsets, table_bucket_offsets=oidx.table_bucket_offsets,
        hash_a=A, hash_b=B, n_total_candidates=len(oidx.candidate_indices), n_total_buckets=oidx.n_total_buckets,
        n_hash_tables=L, n_hashes=k, sig_nbytes=oidx.sig_nbytes, n_features=top, seed=0)
    got = core_mod.MinHashCore(L, k, 0).hash(indices, indptr, len(rows), ix)
    assert np.array_equal(got.transpose(1, 0, 2).reshape(len(rows), H), want)
