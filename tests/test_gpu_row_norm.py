"""Mean row norm behind the default window: rows at the edges of a warp, of a CTA's eight rows and of the grid
(592 CTAs), columns at the edges of a warp's load and of a lane's eight loads, against NumPy in float64 (two
summation orders of at most 20,000 terms: 1e-12 relative); infinite and NaN values; and which rows take it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,d", [(1, 1), (7, 31), (8, 32), (9, 33), (1184, 5), (1185, 100), (10_000, 128), (3, 1000),
                                 (4736, 223), (4737, 224), (5, 225), (5, 255), (6, 256), (7, 257), (2, 20_000)])
def test_equals_numpy(n, d, dtype):
    import torch
    from culsh_b200._culsh_core import mean_row_norm
    X = (5 * np.random.default_rng(n).standard_normal((n, d))).astype(dtype)
    want = np.linalg.norm(X.astype(np.float64), axis=1).mean()
    for _ in range(2):
        assert abs(mean_row_norm(torch.from_numpy(X).cuda()) - want) <= 1e-12 * want


def test_window_of_a_side_stream_and_of_a_strided_view():
    import torch
    from culsh_b200 import PStableLSH
    X = torch.randn(5000, 64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    want = int(torch.linalg.norm(X.double(), dim=1).mean())
    assert PStableLSH._estimate_window_size(X) == want
    wide = torch.randn(5000, 128, device="cuda")
    assert PStableLSH._estimate_window_size(wide[:, ::2]) == int(torch.linalg.norm(wide[:, ::2].double(), dim=1).mean())
    with torch.cuda.stream(torch.cuda.Stream()):
        Y = X
        for _ in range(50):  # work that is still on its way when the window is asked for
            Y = Y * 1.0
        Y = Y * 3.0
        assert PStableLSH._estimate_window_size(Y) == int(torch.linalg.norm(Y.double(), dim=1).mean())


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_values_that_are_not_finite(dtype):
    import torch
    from culsh_b200._culsh_core import mean_row_norm
    X = np.ones((300, 33), dtype)
    X[299, 32] = np.inf
    assert mean_row_norm(torch.from_numpy(X).cuda()) == np.inf
    X[0, 0] = np.nan
    assert np.isnan(mean_row_norm(torch.from_numpy(X).cuda()))
    X = np.full((4, 7), np.finfo(np.float32).max, dtype)  # the squares need float64
    want = np.linalg.norm(X.astype(np.float64), axis=1).mean()
    assert abs(mean_row_norm(torch.from_numpy(X).cuda()) - want) <= 1e-12 * want


def test_which_rows_the_engine_takes(monkeypatch):
    import torch
    from culsh_b200 import PStableLSH, pstable_lsh
    calls = []
    monkeypatch.setattr(pstable_lsh, "mean_row_norm", lambda x: calls.append(x.shape) or 3.0)
    f32, f64 = torch.float32, torch.float64
    for rows, d, dtype, engine in [(1024, 63, f32, True), (1025, 63, f32, False), (1025, 255, f32, False), (1025, 256, f32, True),
                                   (50, 4096, f32, True), (50, 4097, f32, False), (50, 63, f64, False), (2000, 511, f64, False)]:
        X = torch.ones((rows, d), device="cuda", dtype=dtype)
        calls.clear()
        assert PStableLSH._estimate_window_size(X) == (3 if engine else int(np.sqrt(d)))
        assert bool(calls) == engine


def test_cuda_view_of_pinned_memory():
    """torch makes a CUDA tensor of a page-locked buffer that says it is device memory."""
    import torch
    from culsh_b200 import PStableLSH
    from culsh_b200._culsh_core import mean_row_norm
    host = torch.randn(300, 40).mul_(3.0).pin_memory()

    class View:
        __cuda_array_interface__ = {"shape": (300, 40), "typestr": "<f4", "data": (host.data_ptr(), False), "version": 3}

    X = torch.as_tensor(View(), device="cuda")
    if X.data_ptr() != host.data_ptr():
        pytest.skip("this torch copies such a view")
    want = float(torch.linalg.norm(host.double(), dim=1).mean())
    assert abs(mean_row_norm(X) - want) <= 1e-12 * want
    assert PStableLSH(4, 4, seed=1).fit(X).window_size == int(want)


def test_pageable_memory_is_refused():
    import ctypes
    from culsh_b200 import _lib
    from culsh_b200._culsh_core import get_handle
    X, out = np.ones((4, 4), np.float32), ctypes.c_double()
    h = get_handle()
    assert h.lib.culsh_mean_row_norm(h.ptr, X.ctypes.data, 4, 4, 0, ctypes.byref(out)) != 0


@pytest.mark.parametrize("n,d,double,engine", [(4095, 63, False, False), (4096, 63, False, True), (4096, 63, True, True), (4095, 511, True, False),
                                               (4096, 4097, False, False)])
def test_many_rows_go_to_the_engine(n, d, double, engine, monkeypatch):
    import torch
    from culsh_b200 import PStableLSH, pstable_lsh
    calls = []
    monkeypatch.setattr(pstable_lsh, "mean_row_norm", lambda x: calls.append(x.shape) or 3.0)
    PStableLSH._estimate_window_size(torch.ones((n, d), device="cuda", dtype=torch.float64 if double else torch.float32))
    assert bool(calls) == engine
