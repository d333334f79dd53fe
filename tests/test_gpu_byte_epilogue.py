"""One-byte p-stable keys of 2, 4, 8 and 16 hashes are quantised by an add that leaves the floor in the low bits of the sum;
where a sum of a warp's rows is outside a byte, or no number, its columns are quantised by conversions.  Rows whose sums are
at both ends of the byte and beyond, infinite or NaN, in fits (one byte is wide enough, or the next form of the keys is
taken) and in queries (a row outside the index's range is in no bucket), for whole and cut groups of
sixteen columns.  The full-width signatures of the same rows come from the general epilogue and the same sums, so
that everything has to agree."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VALUES = [0.0, -0.0, 1.0, -1.0, 100.0, 126.0, -126.0, 127.0, -127.0, 128.0, -128.0, 129.0, -129.0, 1e4, -1e4, 4e6, -5e6, 1e7, -1e7, 3e9, -3e9,
          1e30, -1e30, np.inf, -np.inf, np.nan]


def _rows(n, seed, values):
    rng = np.random.default_rng(seed)
    X = np.zeros((n, 8), np.float32)
    X[:, 0] = rng.integers(-20, 20, n)
    X[rng.permutation(n)[:len(values)], 0] = values
    return X


@pytest.mark.parametrize("L,k", [(3, 2), (16, 2), (5, 4), (1, 8), (3, 8), (16, 8), (34, 8), (3, 16)])
@pytest.mark.parametrize("n", [1, 127, 129, 700])
@pytest.mark.parametrize("values", [[], [3.0], VALUES])
def test_equals_the_full_width(L, k, n, values):
    from culsh_b200 import _culsh_core as core_mod
    special = VALUES
    if k == 16:
        # Full-width keys of 64 bytes take the kernel of the CUDA cores: its sums round differently once in 200,000,
        # and an infinite row, of which the split makes no number, keeps its sums there.
        n = min(n, 129)
        values, special = ([v for v in vs if not np.isinf(v)] for vs in (values, VALUES))
    X = _rows(n, L * k, np.array(values[:n], np.float32))
    Q = _rows(300, 7, np.array(special, np.float32))
    core = core_mod.PSLSHCore(L, k, 1, 5)
    ix = core.fit_float(X, n, 8)
    sx, sq = core.hash(X, ix), core.hash(Q, ix)  # [L][n][k]
    cand, tab, off = ix.get_candidate_indices(), ix.get_table_bucket_offsets(), ix.get_bucket_candidate_offsets()
    keys = ix.get_bucket_signatures().view(np.int32).reshape(-1, k)
    for t in range(L):
        per_row = np.repeat(keys[tab[t]:tab[t + 1]], np.diff(off[tab[t]:tab[t + 1] + 1]), axis=0)
        assert np.array_equal(per_row, sx[t][cand[t * n:(t + 1) * n]])
    got = core.query_float(Q, 300, ix)
    qo, qi = got.get_offsets().astype(np.int64), got.get_indices()
    for i in range(300):
        hit = (sx == sq[:, i:i + 1]).all(axis=2).any(axis=0)
        assert np.array_equal(qi[qo[i]:qo[i + 1]], np.flatnonzero(hit))
