"""The kernel for float32 rows off 16-byte boundaries has to give the sums of the plain kernel to the last
bit.  A table of more than 128 hashes takes the plain one, and one seed makes the same H x d
projection for L = 1, k = H as for any other split of H, so the signs can be compared one by one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,L,k", [(1, 1, 3, 44), (127, 15, 2, 66), (128, 17, 22, 6), (129, 33, 5, 30), (40_001, 50, 13, 11),
                                     (20_000, 101, 66, 2), (300, 7, 130, 1), (5000, 255, 2, 128),
                                     (40_001, 17, 4, 11), (38_017, 50, 8, 8)])
def test_signs_equal_the_plain_kernel(n, d, L, k):
    from culsh_b200 import _culsh_core as core_mod
    H = L * k
    X = np.random.default_rng(n + d).standard_normal((n, d)).astype(np.float32)
    core = core_mod.RPLSHCore(L, k, 9)
    plain = core_mod.RPLSHCore(1, H, 9)
    tiny = np.ones((1, d), np.float32)
    ix, ix1 = core.fit_float(tiny, 1, d), plain.fit_float(tiny, 1, d)
    assert np.array_equal(ix.get_projection_matrix(), ix1.get_projection_matrix())
    got = core.hash(X, ix).transpose(1, 0, 2).reshape(n, H)
    want = plain.hash(X, ix1).transpose(1, 0, 2).reshape(n, H)
    assert np.array_equal(got, want)
    fit = core.fit_float(X, n, d)  # and the packed keys of a fit are these bits
    cand, tab, off = fit.get_candidate_indices(), fit.get_table_bucket_offsets(), fit.get_bucket_candidate_offsets()
    keys = fit.get_bucket_signatures().reshape(-1, k)
    for t in range(L):
        per_row = np.repeat(keys[tab[t]:tab[t + 1]], np.diff(off[tab[t]:tab[t + 1] + 1]), axis=0)
        assert np.array_equal(per_row, got.reshape(n, L, k)[cand[t * n:(t + 1) * n], t])


@pytest.mark.parametrize("n,d,L,k", [(40_001, 17, 4, 8), (38_017, 50, 8, 8), (40_001, 33, 28, 8), (2_000, 30, 300, 8)])
def test_p_stable_rows_of_later_blocks(n, d, L, k):
    """A CTA that stays gets the same values for the rows of its later blocks as for the same rows in its first one."""
    from culsh_b200 import _culsh_core as core_mod
    X = np.random.default_rng(n + d).standard_normal((n, d)).astype(np.float32)
    core = core_mod.PSLSHCore(L, k, 1, 9)
    ix = core.fit_float(X[:1], 1, d)
    got = core.hash(X, ix)
    for r0 in (0, 127, n // 2, n - 300, n - 100):
        assert np.array_equal(got[:, r0:r0 + 300], core.hash(np.ascontiguousarray(X[r0:r0 + 300]), ix))


def test_many_groups_of_columns():
    """33 groups of 128 columns do not fill the places for CTAs that stay: a CTA for each block and group."""
    from culsh_b200 import _culsh_core as core_mod
    n, d, L, k = 700, 17, 66, 64
    X = np.random.default_rng(5).standard_normal((n, d)).astype(np.float32)
    core = core_mod.RPLSHCore(L, k, 9)
    ix = core.fit_float(X, n, d)
    P = ix.get_projection_matrix().reshape(L * k, d).astype(np.float64)
    S = X.astype(np.float64) @ P.T
    got = core.hash(X, ix).transpose(1, 0, 2).reshape(n, L * k)
    clear = np.abs(S) > 17 * 2.0**-23 * (np.abs(X) @ np.abs(P).T)  # beyond the rounding of a sum of 17 terms
    assert clear.mean() > 0.999 and np.array_equal(got[clear], (S > 0)[clear])
