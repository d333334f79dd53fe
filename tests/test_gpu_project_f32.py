"""The kernel for float32 rows off 16-byte boundaries has to give the sums of the plain kernel to the last
bit.  A table of more than 128 hashes takes the plain one, and one seed makes the same H x d
projection for L = 1, k = H as for any other split of H, so the signs can be compared one by one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,L,k", [(1, 1, 3, 44), (127, 15, 2, 66), (128, 17, 22, 6), (129, 33, 5, 30), (40_001, 50, 13, 11),
                                     (20_000, 101, 66, 2), (300, 7, 130, 1), (5000, 255, 2, 128)])
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
