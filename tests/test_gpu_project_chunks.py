"""P-stable keys of one-byte elements with 2, 4 or 8 hashes are packed by a form of their own, in steps of
sixteen columns, by two groups of warps that share the tables of a chunk: odd numbers of tables in a chunk, last
chunks that are shorter, and one table.  The signatures of `hash` take the general form over the
same sums, so that every byte has to agree."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,k", [(1, 8), (3, 8), (13, 8), (17, 8), (33, 8), (34, 8), (42, 8), (7, 4), (66, 4), (67, 4), (5, 2),
                                 (33, 2), (131, 2), (130, 1), (34, 6)])
@pytest.mark.parametrize("n,d", [(130, 32), (300, 100)])
def test_fit_keys_equal_signatures(n, d, L, k):
    from culsh_b200 import _culsh_core as core_mod
    X = np.random.default_rng(L * k).standard_normal((n, d)).astype(np.float32)
    core = core_mod.PSLSHCore(L, k, 4, 11)
    ix = core.fit_float(X, n, d)
    sig = core.hash(X, ix)  # [L][n][k]
    assert core.last_stats()["hash_path"] == 1
    cand, tab, off = ix.get_candidate_indices(), ix.get_table_bucket_offsets(), ix.get_bucket_candidate_offsets()
    keys = np.ascontiguousarray(ix.get_bucket_signatures()).reshape(ix.n_total_buckets, -1).view(np.int32)
    for t in range(L):
        per_row = np.repeat(keys[tab[t]:tab[t + 1]], np.diff(off[tab[t]:tab[t + 1] + 1]), axis=0)
        assert np.array_equal(per_row, sig[t][cand[t * n:(t + 1) * n]])
    c = core.query_float(X, n, ix)  # query keys come with their range flags
    at, ids = c.get_offsets().astype(np.int64), c.get_indices()
    assert all(i in ids[at[i]:at[i + 1]] for i in range(0, n, 17))
