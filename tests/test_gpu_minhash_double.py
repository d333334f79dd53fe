"""MinHash rows of column ids below 2^20 are hashed with double-precision multiply-adds: ids on both sides of the line, alone,
in odd and even numbers and mixed inside one 32-id step, for every number of hash functions per lane, with parameters at the
ends of their range (the largest product and sum there are) and values next to the prime, against the 64-bit oracle."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,k", [(4, 1), (8, 7), (12, 8), (16, 8), (20, 8), (24, 8), (28, 8), (32, 8), (40, 9)])
def test_columns_around_the_double_line(L, k):
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(L)
    line, top = 1 << 20, (1 << 22) - 1
    rows = [[line - 1], [line], [0], [0, line - 1], [0, line - 1, line], [], list(range(line - 40, line + 40)), list(range(line - 40, line)),
            [0] * 31 + [top], sorted(rng.integers(0, line, 33)), sorted(rng.integers(0, line, 64)), sorted(rng.integers(0, line, 65)),
            sorted(rng.integers(0, top, 200)), list(range(32)) + [top - 1], list(range(31)), [line - 1] * 3]
    H, p = L * k, oracle.MINHASH_PRIME
    A = rng.integers(1, p, H).astype(np.uint32)
    B = rng.integers(0, p, H).astype(np.uint32)
    A[-1] = B[-1] = p - 1      # the largest sum
    A[0], B[1] = 1, 0
    for h, (c, v) in enumerate([(line - 1, p - 1), (line, p - 1), (0, p - 5), (line - 1, 0)][:H - 1]):
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
