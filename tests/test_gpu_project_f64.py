"""float64 projection on the matrix instructions: rows, features and hash columns on both sides of the
64-row tile, the 16-feature stage, the 8-column step and the 128-column group, CTAs that stay for several
blocks of rows and shapes past the lines where they do not, against the CUDA-core kernel (projection
path 1).  Both round in float64: a sign or floor may differ only where the sum lies
within d * 2^-52 * sum|x p| of the boundary, which for standard normals and a few million values
happens with a probability below 1e-6, so the signatures are compared whole."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family", ["rplsh", "pslsh"])
@pytest.mark.parametrize("n,d,L,k", [(1, 1, 2, 1), (63, 14, 2, 4), (64, 30, 3, 5), (65, 31, 2, 16), (127, 15, 2, 4), (128, 16, 1, 8), (129, 17, 3, 6), (300, 32, 16, 8),
                                     (300, 33, 17, 8), (513, 50, 2, 9), (260, 100, 16, 14), (200, 7, 2, 15), (64, 256, 130, 1),
                                     (38_001, 17, 4, 8), (20_500, 47, 8, 8), (20_500, 50, 2, 16), (9_501, 33, 28, 8), (20_500, 100, 8, 8), (2_000, 20, 300, 8), (700, 17, 264, 16)])
def test_equals_cuda_core_projection(family, n, d, L, k):
    from culsh_b200 import _culsh_core as core_mod
    X = np.random.default_rng(n * d).standard_normal((n, d))
    core = core_mod.RPLSHCore(L, k, 5) if family == "rplsh" else core_mod.PSLSHCore(L, k, 2, 5)
    try:
        ix = core.fit_double(X, n, d)
        sig = core.hash(X, ix)
        keys, cand = ix.get_bucket_signatures(), ix.get_candidate_indices()
        core.set_projection_path(1)
        ix1 = core.fit_double(X, n, d)
        assert np.array_equal(sig, core.hash(X, ix1))
        assert np.array_equal(keys, ix1.get_bucket_signatures())
        assert np.array_equal(cand, ix1.get_candidate_indices())
    finally:
        core.set_projection_path(0)
