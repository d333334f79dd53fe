"""Batches of a query share their launches as long as their lists are few, and the scans of a batch run in
one CTA up to 32,768 queries: query counts at the edges of the scan's 4096-element steps and of that line, batch
sizes that leave a rest, and lists of more than 2^25 entries, which are taken batch by batch, have to give
what one batch gives (tests/test_query_groups.py has the way back when memory is short).  P-stable fits keep the range of their hash values on the way: bytes at the edges of
the compressed sort (32 levels) and of the byte itself, in each projection kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b):
    for f in ("get_indices", "get_offsets", "get_counts"):
        assert np.array_equal(getattr(a, f)(), getattr(b, f)())


@pytest.mark.parametrize("nq,batch", [(4095, 1000), (4096, 4095), (4097, 64), (8191, 1000), (8192, 8191), (8193, 64), (32_767, 32_766), (32_768, 5000), (32_769, 16_384)])
def test_query_counts(nq, batch):
    import culsh_b200 as culsh
    rng = np.random.default_rng(nq)
    X = rng.standard_normal((20_000, 16)).astype(np.float32)
    Q = rng.standard_normal((nq, 16)).astype(np.float32)
    m = culsh.RPLSH(6, 14, seed=2).fit(X)
    _same(m.query(Q, batch_size=batch), m.query(Q))


def test_long_lists_go_batch_by_batch():
    import culsh_b200 as culsh
    rng = np.random.default_rng(0)
    X = rng.standard_normal((100_000, 8)).astype(np.float32)
    m = culsh.RPLSH(4, 2, seed=2).fit(X)
    Q = rng.standard_normal((501, 8)).astype(np.float32)  # about 4 x 25,000 entries each: 2^25.6
    _same(m.query(Q, batch_size=100), m.query(Q))


@pytest.mark.parametrize("dtype,d,k", [(np.float32, 8, 8), (np.float32, 8, 5), (np.float32, 7, 4), (np.float64, 8, 8)])
@pytest.mark.parametrize("scale", [0.3, 3.0, 4.5, 12.0, 40.0])
def test_hash_value_range(dtype, d, k, scale):
    from culsh_b200 import _culsh_core as core_mod
    n, L = 5000, 3
    X = (scale * np.random.default_rng(d).standard_normal((n, d))).astype(dtype)
    core = core_mod.PSLSHCore(L, k, 1, 3)
    ix = (core.fit_float if dtype == np.float32 else core.fit_double)(X, n, d)
    sig = core.hash(X, ix)  # [L][n][k] at full width
    cand = ix.get_candidate_indices()
    for t in range(L):
        raw = np.ascontiguousarray(sig[t]).view(np.uint8).reshape(n, 4 * k)
        order = np.lexsort(tuple(raw[:, j] for j in range(4 * k - 1, -1, -1)))
        assert np.array_equal(cand[t * n:(t + 1) * n], order)


def test_more_pairs_than_fit_30_bits():
    """A query without batches above 2^30 (table, query) pairs, against the same one in batches."""
    import torch
    import culsh_b200 as culsh
    from culsh_b200._culsh_core import MinHashCore
    n, L, nq = 2000, 1024, (1 << 20) + 3
    g = torch.Generator("cuda").manual_seed(3)
    X = torch.randn(n, 8, device="cuda", generator=g)
    Q = torch.randn(nq, 8, device="cuda", generator=g)
    Q[::1000] = X[:1049]
    m = culsh.RPLSH(L, 30, seed=2).fit(X)
    whole, parts = m.query(Q), m.query(Q, batch_size=300_000)
    assert torch.equal(whole.get_indices(as_torch=True), parts.get_indices(as_torch=True))
    assert torch.equal(whole.get_offsets(as_torch=True).view(torch.int64), parts.get_offsets(as_torch=True).view(torch.int64))
    assert whole.n_total_candidates >= 1049
    del whole, parts, m, Q
    ids = torch.randint(0, 1 << 28, (2 * nq,), device="cuda", generator=g, dtype=torch.int32)
    ptr = (2 * torch.arange(nq + 1, device="cuda")).to(torch.int32)
    core = MinHashCore(L, 2, 5)
    ix = core.fit(ids[:2 * n], ptr[:n + 1].contiguous(), n, 1 << 28)
    c = core.query(ids, ptr, nq, ix)
    off = c.get_offsets()
    few = core.query(ids[:2 * n], ptr[:n + 1].contiguous(), n, ix)
    assert np.array_equal(off[:n + 1], few.get_offsets())
    assert np.array_equal(c.get_indices()[:int(off[n])], few.get_indices())
    core.trim_scratch(0)
