"""The tensor-core gradient at the edges of its tiles: a warp has 16 samples, a block 64,
the grid 304 blocks, whose next tile is loaded ahead.  Against the oracle's gradient, with the
bounds of the two-term BF16 signals (about 16 bits): loss 1e-5, gradient 1e-4 of its norm."""
import numpy as np
import pytest

from oracle import indicator_oracle as IO
from test_gpu_indicator import model_with, random_net

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 17, 64, 65, 304 * 64 - 1, 304 * 64 + 1])
def test_gradient_tile_edges(gpu_lib, n):
    import torch
    p, norm, X, y = random_net(5, 2 * n + 64)
    _, prone = IO.forward_tensor_core(p, norm, X)
    X, y = (np.ascontiguousarray(v[~prone][:n]) for v in (X, y))
    assert len(X) == n
    m = model_with(p, norm)
    loss, g = m.gradient(torch.from_numpy(X).cuda(), torch.from_numpy(y).cuda(), 3.0)
    lo, go = IO.loss_and_grad(p, norm, X, y, 3.0, tensor_core=True)
    assert abs(loss - lo) <= 1e-5 * abs(lo)
    assert np.linalg.norm(g - go) <= 1e-4 * np.linalg.norm(go)
