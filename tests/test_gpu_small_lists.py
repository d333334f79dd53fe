"""Lists of more than four ids are fetched end to end by the warp of their query, in a self-join one after another: rows in
groups of equal ones, so that every list of a query holds its group, below and above four ids, for numbers of tables on both
sides of a warp's 32 and 64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [1, 31, 32, 33, 64, 65, 100])
@pytest.mark.parametrize("sizes", [(4, 5), (1, 4, 6, 40), (5, 33, 90)])
def test_lists_of_all_lengths(L, sizes):
    """Rows in groups of equal ones: every list of a query holds its group, below and above four ids."""
    import culsh_b200 as culsh
    rng = np.random.default_rng(L)
    base = rng.standard_normal((400, 12)).astype(np.float32)
    group = np.repeat(np.arange(400), [sizes[i % len(sizes)] for i in range(400)])
    group = group[rng.permutation(len(group))]
    X = base[group]
    lsh = culsh.RPLSH(L, 30, seed=5)
    m = lsh.fit(X)
    for cand, queries in ((m.query(np.repeat(base, 20, axis=0)), np.repeat(np.arange(400), 20)), (lsh.fit_query(X), group)):
        off, ids = cand.get_offsets().astype(np.int64), cand.get_indices()
        for i in rng.integers(0, len(queries), 500):
            assert set(np.flatnonzero(group == queries[i])) <= set(ids[off[i]:off[i + 1]])
            assert np.all(np.diff(ids[off[i]:off[i + 1]]) > 0)
    want = m.query(X)
    got = lsh.fit_query(X)
    assert np.array_equal(want.get_indices(), got.get_indices()) and np.array_equal(want.get_offsets(), got.get_offsets())
