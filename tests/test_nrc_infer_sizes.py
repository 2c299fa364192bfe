"""Inference at the sizes where its tiles end: a lone sample, the edges of a
128-sample tile, a tile for each group of each block and one more or less,
several rounds -- a sample's output does not depend on where in a call it
stands, so a call equals the calls of its pieces exactly; and the outputs
stay within the buffer."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ROUND = 152 * 3 * 128


@pytest.mark.parametrize("n", [1, 127, 128, 129, 383, 385, ROUND - 128, ROUND - 1, ROUND, ROUND + 1, 2 * ROUND + 129, 3 * ROUND - 5])
def test_call_equals_its_pieces(gpu_lib, n):
    cache = gpu_lib.RadianceCache(seed=3)
    x = torch.tensor(np.random.default_rng(n).normal(size=(n, 9)).astype(np.float32), device="cuda")
    y = torch.full((n + 1, 3), 7.0, device="cuda")
    cache.infer(x, y[:n])
    assert (y[n] == 7.0).all()
    piece = max(1, n // 5 + 37)
    z = torch.empty(n, 3, device="cuda")
    for a in range(0, n, piece):
        part = x[a:a + piece].clone()
        out = torch.empty(part.shape[0], 3, device="cuda")
        cache.infer(part, out)
        z[a:a + piece] = out
    assert torch.equal(y[:n], z)
