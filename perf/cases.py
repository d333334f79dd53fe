"""Performance cases of the LSH engine: what its users have it do, through the public entry
points, from one query against a kept index up to the self-join of ten million rows.

A case is a dict of plain values:

  family  rplsh | pslsh | minhash
  mode    fit+query   index n rows, then look nq queries up (a fresh index on every pass)
          query       look nq queries up in an index that the program keeps
          fit_query   self-join: index n rows and look every one of them up
  n, nq   rows and queries; nq is 0 for a self-join
  d       columns (MinHash: size of the column-id universe)
  L, k    hash tables and hashes per table
  w       p-stable bucket width, 0 for the default "auto"; 0 for the other families
  f64     float64 rows instead of float32
  host    the program holds NumPy / SciPy data and wants NumPy results; otherwise everything
          stays on the GPU
  batch   query batch size, 0 for none
  law     value law of the rows:
            counts   non-negative integers with a heavy tail, as image descriptors have
            sphere   points of the unit sphere
            normal   independent standard normals
            mixture  4,096 Gaussian clusters (spread 0.15)
            zipf     CSR rows of lo..hi column ids, Zipf-distributed (exponent 1.1)
  lo, hi  row lengths of the CSR rows (0 for dense rows)
"""
import math

import numpy as np
import torch

import culsh_b200
from culsh_b200 import minhash_lsh
from culsh_b200._culsh_core import MinHashCore

LSH_SEED = 42  # a program keeps one configuration, seed included, for all the data it indexes


def _case(name, family, mode, n, nq, d, L, k, law, w=0, f64=False, host=False, batch=0, lo=0, hi=0):
    c = dict(family=family, mode=mode, n=n, nq=nq, d=d, L=L, k=k, w=w, f64=f64, host=host, batch=batch,
             law=law, lo=lo, hi=hi)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one query of an online service against a kept index of a million descriptors
        _case("rplsh_one_query", "rplsh", "query", 1_000_000, 1, 128, 32, 16, "counts"),
        # near duplicates inside a small batch of vectors, all defaults
        _case("pslsh_tiny_self_join", "pslsh", "fit_query", 1_000, 0, 100, 8, 8, "normal"),
        # a small collection indexed and queried at once; the window comes from the data
        _case("pslsh_small", "pslsh", "fit+query", 10_000, 100, 128, 16, 8, "normal"),
        # the benchmark's million descriptors with ten thousand queries
        _case("rplsh_million", "rplsh", "fit+query", 1_000_000, 10_000, 128, 32, 16, "counts"),
        # offline lookup of many queries in the batches the examples use, short candidate lists
        _case("rplsh_batched_lookup", "rplsh", "query", 1_000_000, 100_003, 96, 24, 18, "sphere", batch=10_000),
        # a NumPy program: rows and queries in ordinary host memory, candidates wanted there
        _case("rplsh_numpy", "rplsh", "fit+query", 400_000, 4_000, 128, 32, 16, "counts", host=True),
        # NumPy's default precision, moved to the GPU by the program
        _case("rplsh_double", "rplsh", "fit+query", 200_003, 2_001, 100, 16, 14, "sphere", f64=True),
        # a width that is not a multiple of four, keys that are not a power of two of bytes
        _case("pslsh_ragged", "pslsh", "fit+query", 333_337, 3_001, 50, 10, 6, "mixture", w=3),
        # near-duplicate documents of a SciPy matrix
        _case("minhash_scipy_self_join", "minhash", "fit_query", 100_003, 0, 1 << 20, 32, 4, "zipf",
              host=True, lo=20, hi=200),
        # two million sets on the GPU with ten thousand queries
        _case("minhash_sets", "minhash", "fit+query", 2_000_000, 10_000, 1 << 20, 32, 4, "zipf", lo=20, hi=200),
        # one GPU's shard of a hundred million vectors
        _case("pslsh_shard", "pslsh", "fit+query", 12_500_000, 10_000, 96, 16, 8, "mixture", w=4),
        # the largest: every near pair of ten million vectors
        _case("rplsh_self_join", "rplsh", "fit_query", 10_000_000, 0, 256, 48, 24, "sphere"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(("rplsh", "pslsh", "minhash"))
    mode = rng.choice(("fit+query", "query", "fit_query"))
    host = rng.random() < 0.25
    if family == "minhash":
        n = _log_int(rng, 1_000, 400_000 if host or mode == "fit_query" else 2_000_000)
        lo = rng.randint(5, 30)
        hi = lo + rng.randint(10, 170)
        L, k, d, law, w, f64 = rng.randint(8, 32), rng.randint(3, 5), 1 << rng.randint(16, 22), "zipf", 0, False
    else:
        lo = hi = 0
        f64 = rng.random() < 0.2
        n = _log_int(rng, 1_000, 1_000_000 if host or f64 else 5_000_000)
        d = _log_int(rng, 24, 256)
        if rng.random() < 0.5:
            d = max(4, d // 4 * 4)
        if family == "rplsh":
            # about log2(n) sign bits keep the buckets short, a few less for rows that spread evenly
            L, w = rng.randint(8, 40), 0
            law = rng.choice(("counts", "sphere")) if mode != "fit_query" else "sphere"
            k = max(8, int(round(math.log2(n))) + rng.randint(-3, 2)) if law == "sphere" else max(8, int(round(math.log2(n))) - rng.randint(2, 4))
        else:
            L, k = rng.randint(8, 16), rng.randint(6, 10)
            law = "normal" if n <= 10_000 else "mixture"
            # the default looks at the data; a width of its own follows the spread of the projections
            w = 0 if law == "normal" else max(1, int(round(0.4 * math.sqrt(d))))
        L += L % 2  # single-precision and double parameters come in pairs: L * k * d has to be even
    nq = 0 if mode == "fit_query" else _log_int(rng, 1, 10_000 if mode == "fit+query" or family == "minhash" else 50_000)
    if law == "counts":  # a query finds about a fiftieth of the rows: bound the ids of a pass
        nq = min(nq, max(1, 10_000_000_000 // n))
    batch = 10_000 if family != "minhash" and nq > 10_000 and rng.random() < 0.5 else 0
    return _case(None, family, mode, n, nq, d, L, k, law, w, f64, host, batch, lo, hi)


# ------------------------------------------------------------------------------------------
# inputs: one collection for each case; the seed sets the order of its rows and queries, so that
# every row id is another one while the number of candidates stays
# ------------------------------------------------------------------------------------------
def _rows(c, n, g, centres):
    d, law = c["d"], c["law"]
    if law == "counts":
        x = torch._standard_gamma(torch.full((n, d), 0.5, device="cuda"), generator=g)
        return x.mul_(40.0).round_().clamp_(0, 255)
    if law == "mixture":
        x = torch.randn(n, d, device="cuda", generator=g).mul_(0.15)
        at = torch.randint(0, centres.shape[0], (n,), device="cuda", generator=g)
        for r0 in range(0, n, 1 << 20):  # in pieces: no second array of this size
            x[r0:r0 + (1 << 20)] += centres[at[r0:r0 + (1 << 20)]]
        return x
    x = torch.randn(n, d, device="cuda", generator=g)
    return x.div_(x.norm(dim=1, keepdim=True)) if law == "sphere" else x


def _dense(c, seed):
    """Rows, and queries of which half are indexed rows with a tenth of noise and half are new."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    centres = torch.randn(4096, c["d"], device="cuda", generator=g) if c["law"] == "mixture" else None
    X, Q = _rows(c, c["n"], g, centres), None
    if c["nq"]:
        Q = _rows(c, c["nq"], g, centres)
        old = (c["nq"] + 1) // 2
        src = X[torch.randint(0, c["n"], (old,), device="cuda", generator=g)]
        noise = 0.1 * src.std(dim=1, keepdim=True) * torch.randn(old, c["d"], device="cuda", generator=g)
        Q[:old] = (src + noise).round_().clamp_(0, 255) if c["law"] == "counts" else src + noise
    if c["f64"]:
        # values that a float32 cannot hold, as measured data in float64 has
        X, Q = (None if x is None else x.double().mul_(1.0 + 1e-9 * math.pi) for x in (X, Q))
    g.manual_seed(seed)
    X = X[torch.randperm(c["n"], device="cuda", generator=g)]
    return X, None if Q is None else Q[torch.randperm(c["nq"], device="cuda", generator=g)]


def _zipf(c, count, g):
    u = torch.rand(count, device="cuda", generator=g, dtype=torch.float64)
    a = -0.1
    x = (1.0 - u * (1.0 - float(c["d"]) ** a)) ** (1.0 / a)
    return (x.to(torch.int64) - 1).clamp_(0, c["d"] - 1)


def _csr(rows, cols, n):
    key = torch.unique((rows << 32) | cols)  # sorted rows without repeated ids
    indptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    indptr[1:] = torch.cumsum(torch.bincount(key >> 32, minlength=n), 0)
    return (key & 0xFFFFFFFF).to(torch.int32), indptr.to(torch.int32)


def _take(csr, which):
    """(row number in the result, ids) of the rows `which` of a CSR matrix."""
    indices, indptr = csr
    first, size = indptr[which].long(), (indptr[which + 1] - indptr[which]).long()
    rows = torch.repeat_interleave(torch.arange(len(which), device="cuda"), size)
    at = torch.arange(int(rows.numel()), device="cuda") - torch.repeat_interleave(size.cumsum(0) - size - first, size)
    return rows, indices[at], size


def _reorder(csr, n, g):
    _, indices, size = _take(csr, torch.randperm(n, device="cuda", generator=g))
    indptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    indptr[1:] = size.cumsum(0)
    return indices.contiguous(), indptr.to(torch.int32)


def _new_sets(c, n, g):
    size = torch.randint(c["lo"], c["hi"] + 1, (n,), device="cuda", generator=g)
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), size)
    return rows, _zipf(c, int(rows.numel()), g)


def _sets(c, seed):
    """Sets, and queries of which half are indexed sets with a tenth of the ids replaced."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    X, Q = _csr(*_new_sets(c, c["n"], g), c["n"]), None
    if c["nq"]:
        old = (c["nq"] + 1) // 2
        rows, cols, _ = _take(X, torch.randint(0, c["n"], (old,), device="cuda", generator=g))
        swap = torch.rand(rows.numel(), device="cuda", generator=g) < 0.1
        cols = torch.where(swap, _zipf(c, int(rows.numel()), g), cols.long())
        new_rows, new_cols = _new_sets(c, c["nq"] - old, g)
        Q = _csr(torch.cat([rows, new_rows + old]), torch.cat([cols, new_cols]), c["nq"])
    g.manual_seed(seed)
    X = _reorder(X, c["n"], g)
    return X, None if Q is None else _reorder(Q, c["nq"], g)


def _scipy(c, csr, n):
    indices, indptr = (x.cpu().numpy() for x in csr)
    return minhash_lsh.scipy.sparse.csr_matrix((np.ones(len(indices), np.int8), indices, indptr), shape=(n, c["d"]))


def _lsh(c):
    if c["family"] == "rplsh":
        return culsh_b200.RPLSH(c["L"], c["k"], seed=LSH_SEED)
    if c["family"] == "pslsh":
        return culsh_b200.PStableLSH(c["L"], c["k"], window_size=c["w"] or "auto", seed=LSH_SEED)
    return culsh_b200.MinHashLSH(c["L"], c["k"], seed=LSH_SEED)


def prepare(case, seed):
    c = case
    X, Q = (_sets if c["family"] == "minhash" else _dense)(c, seed)
    lsh = _lsh(c)
    if c["family"] == "minhash":
        if c["host"]:
            X, Q = _scipy(c, X, c["n"]), None if Q is None else _scipy(c, Q, c["nq"])
        else:  # sets that are on the GPU already go in as their two arrays
            lsh = MinHashCore(c["L"], c["k"], LSH_SEED)
    elif c["host"]:
        X, Q = X.cpu().numpy(), None if Q is None else Q.cpu().numpy()
    state = dict(case=c, lsh=lsh, X=X, Q=Q, model=None)
    if c["mode"] == "query":
        torch.cuda.synchronize()
        state["model"] = _fit(state)
        state["X"] = None
    return state


def _fit(state):
    c, X = state["case"], state["X"]
    if isinstance(state["lsh"], MinHashCore):
        return state["lsh"].fit(X[0], X[1], c["n"], c["d"])
    return state["lsh"].fit(X)


def _query(state, model):
    c, Q = state["case"], state["Q"]
    if isinstance(state["lsh"], MinHashCore):
        return state["lsh"].query(Q[0], Q[1], c["nq"], model)
    if c["family"] == "minhash":
        return model.query(Q)
    return model.query(Q, batch_size=c["batch"] or None)


def run(state):
    c, X = state["case"], state["X"]
    if c["mode"] == "fit_query":
        if isinstance(state["lsh"], MinHashCore):
            cand = state["lsh"].fit_query(X[0], X[1], c["n"], c["d"])
        else:
            cand = state["lsh"].fit_query(X)
    else:
        cand = _query(state, state["model"] or _fit(state))
    if c["host"]:
        return {"ids": cand.get_indices(), "offsets": cand.get_offsets()}
    return {"ids": cand.get_indices(as_torch=True), "offsets": cand.get_offsets(as_torch=True).view(torch.int64)}


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------
def _ids_out(c):
    """Candidate ids of one pass, fitted to what the laws give: a query finds its own row or
    cluster, and what chance puts into its buckets."""
    q = c["nq"] or c["n"]
    if c["family"] == "minhash":
        return q * (1.0 + c["n"] * c["L"] * 0.1 ** c["k"])
    if c["law"] == "counts":  # all rows lie in one orthant: buckets are far from even
        return q * c["n"] * (1.0 - math.exp(-c["L"] * 0.625 ** c["k"]))
    if c["law"] == "mixture":
        return q * max(1.0, 0.24 * c["n"] / 4096)
    if c["law"] == "normal":
        return q * (1.0 + 4e-4 * c["n"])
    return q * (1.0 + (1.4 + (70.0 / c["d"]) ** 2) * c["L"] * c["n"] / 2.0 ** c["k"])


def work(case):
    """Rows and queries read once, candidates written once, and, where an index is built, its
    row ids written once; flops of the projections (dense) or three integer multiply-adds for
    each (id, hash) pair (MinHash)."""
    c = case
    hashed = c["nq"] + (0 if c["mode"] == "query" else c["n"])
    if c["family"] == "minhash":
        ids = hashed * (c["lo"] + c["hi"]) / 2.0
        read, flops = 4.0 * (ids + hashed), 6.0 * ids * c["L"] * c["k"]
    else:
        read, flops = (8.0 if c["f64"] else 4.0) * hashed * c["d"], 2.0 * hashed * c["d"] * c["L"] * c["k"]
    index = 0.0 if c["mode"] == "query" else 4.0 * c["n"] * c["L"]
    return {"bytes": read + index + 4.0 * _ids_out(c) + 8.0 * (c["nq"] or c["n"]), "flops": flops}


def tolerance(case):
    """Row ids and offsets are whole numbers.  MinHash and the index arithmetic are exact; a
    projection that lies within rounding of a bucket boundary may fall on either side of it in
    another correct implementation, which moves a row in one table."""
    if case["family"] == "minhash":
        return "exact"
    return {"rel": 1e-5, "differ": 1e-3}
