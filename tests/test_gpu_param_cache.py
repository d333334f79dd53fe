"""Hash parameters are kept by the handle.  Configurations of one seed and one L * k have the same
projection matrix but another split of it into chunks for the tensor cores: fits of two of them in turn have to
give the signatures and the index that they give with the cache off.  Pairs whose chunks hold equally many columns,
and pairs of different chunk sizes, in both orders."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, D = 3000, 64


def _fit(core_mod, family, L, k, X):
    core = core_mod.RPLSHCore(L, k, 42) if family == "rplsh" else core_mod.PSLSHCore(L, k, 2, 42)
    ix = core.fit_float(X, N, D)
    return (core.hash(X, ix), ix.get_candidate_indices(), ix.get_bucket_signatures(),
            ix.get_table_bucket_offsets(), ix.get_projection_matrix())


@pytest.mark.parametrize("family,a,b", [
    ("rplsh", (25, 16), (50, 8)), ("rplsh", (50, 8), (25, 16)), ("rplsh", (22, 13), (13, 22)), ("rplsh", (13, 22), (22, 13)),
    ("rplsh", (24, 18), (18, 24)), ("rplsh", (8, 16), (16, 8)), ("pslsh", (20, 14), (40, 7)), ("pslsh", (40, 7), (20, 14)),
])
def test_two_splits_of_one_projection(family, a, b):
    from culsh_b200 import _culsh_core as core_mod
    X = np.random.default_rng(1).standard_normal((N, D)).astype(np.float32)
    switch = core_mod.RPLSHCore(1, 2, 0)
    switch.set_param_cache(False)  # also drops what is kept
    try:
        want = [_fit(core_mod, family, *c, X) for c in (a, b)]
    finally:
        switch.set_param_cache(True)
    for c, w in zip((a, b, a), (want[0], want[1], want[0])):
        for got, exact in zip(_fit(core_mod, family, *c, X), w):
            assert np.array_equal(got, exact)
