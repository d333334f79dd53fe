"""Mean row norm behind the default window: rows at the edges of a warp, of a CTA's eight rows and of the grid,
against NumPy in float64 (two summation orders of at most 10,000 terms: 1e-12 relative)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,d", [(1, 1), (7, 31), (8, 32), (9, 33), (1184, 5), (1185, 100), (10_000, 128), (3, 1000)])
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
