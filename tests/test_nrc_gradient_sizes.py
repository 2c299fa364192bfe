"""The gradient kernel at the sizes where its tiles end: a lone sample, the
edges of a warp's 16 rows and of a block's 128, one and several tiles per
block, and a gradient buffer whose address is only 4-byte aligned -- against
the oracle's bfloat16-rounded backward pass, with the bar of
test_nrc_gpu.py's gradient test (3 % of each parameter block's norm; the
loss 1 %)."""
import numpy as np
import pytest
import torch

from oracle import nrc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 17, 100, 127, 128, 129, 1000, 128 * 152, 128 * 152 + 1, 50001])
@pytest.mark.parametrize("shift", [0, 1])
def test_gradient_by_size(gpu_lib, n, shift):
    rng = np.random.default_rng(n)
    p = nrc.init_params(n % 7)
    p[-3:] = (0.3, 0.4, 0.5)
    x = np.concatenate([rng.uniform(0, 1, (n, 3)), rng.normal(size=(n, 6)) * 0.4], 1).astype(np.float32)
    t = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    cache = gpu_lib.RadianceCache(seed=1)
    cache.set_params(p)
    buf = torch.full((nrc.N_PARAMS + 3,), 7.0, device="cuda")
    grad = buf[shift:shift + nrc.N_PARAMS]
    loss = torch.full((1,), 7.0, device="cuda")
    cache.gradients(torch.tensor(x, device="cuda"), torch.tensor(t, device="cuda"), grad, loss)
    y, c = nrc.forward(p, x)
    ref_loss, dy = nrc.loss_and_dy(y, t)
    ref = nrc.backward(c, dy)
    got = grad.cpu().numpy().astype(np.float64)
    assert abs(loss.item() - ref_loss) <= 1e-2 * ref_loss
    off = 0
    for s in nrc.SHAPES:
        k = int(np.prod(s))
        assert np.linalg.norm(got[off:off + k] - ref[off:off + k]) <= 3e-2 * np.linalg.norm(ref[off:off + k]) + 1e-12
        off += k
    assert (buf[:shift] == 7.0).all() and (buf[shift + nrc.N_PARAMS:] == 7.0).all()
    # a second call starts from nothing; training after it too
    again = torch.empty_like(grad)
    cache.gradients(torch.tensor(x, device="cuda"), torch.tensor(t, device="cuda"), again, loss)
    assert torch.allclose(again, grad.clone(), rtol=1e-3, atol=1e-6 * float(grad.abs().max()) + 1e-12)
