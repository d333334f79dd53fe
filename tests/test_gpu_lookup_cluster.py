"""Few pairs of a table and a query are looked up by one CTA up to 512, by a cluster of eight up to 8,192: numbers of pairs on
both sides of these, queries without a bucket and with long lists among them, against the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,nq", [(1, 1), (1, 512), (1, 513), (2, 256), (2, 257), (16, 32), (16, 33), (3, 1000), (32, 256), (32, 257), (1, 8192),
                                  (1, 8193), (13, 630), (13, 631)])
@pytest.mark.parametrize("family,k", [("rp", 10), ("ps", 5), ("rp", 40)])
def test_candidates_of_the_host(L, nq, family, k):
    from culsh_b200 import _culsh_core as core_mod
    rng = np.random.default_rng(L + nq)
    n, d = 3000, 8
    X = rng.standard_normal((n, d)).astype(np.float32)
    X[rng.random(n) < 0.4] = X[0]  # a bucket of long lists
    Q = X[rng.integers(0, n, nq)].copy()
    far = rng.random(nq) < 0.3
    Q[far] = 50.0 * rng.standard_normal((int(far.sum()), d)).astype(np.float32)
    core = core_mod.RPLSHCore(L, k, 5) if family == "rp" else core_mod.PSLSHCore(L, k, 2, 5)
    ix = core.fit_float(X, n, d)
    rows, qs = core.hash(X, ix), core.hash(Q, ix)
    res = core.query_float(Q, nq, ix)
    ids, off = np.asarray(res.get_indices()), np.asarray(res.get_offsets())
    as_bytes = lambda s: np.ascontiguousarray(s).view(np.uint8).reshape(len(s), -1)
    tables = []
    for t in range(L):
        by = {}
        for i, key in enumerate(map(bytes, as_bytes(rows[t]))):
            by.setdefault(key, []).append(i)
        tables.append(([by.get(bytes(key), []) for key in as_bytes(qs[t])]))
    for q in range(nq):
        want = sorted(set().union(*[tables[t][q] for t in range(L)])) if L else []
        assert np.array_equal(ids[off[q]:off[q + 1]], want)
