"""The MLP training kernel's tile loop (one CTA an SM, a 128-row tile after another): gradients against the numpy oracle
at row counts around one and two tiles per SM.  Tolerance: the BF16-emulating oracle comparison's 5e-3 relative L2."""
import numpy as np
import pytest

from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles, extra", [(1, 0), (1, 1), (2, -1), (2, 77)])
def test_gradient_around_whole_rounds_of_tiles(tiles, extra):
    import torch
    from diffphd_b200.warmstart import WarmStartMLP
    dev = torch.device("cuda:0")
    n = tiles * torch.cuda.get_device_properties(dev).multi_processor_count * 128 + extra
    rng = np.random.default_rng(2)
    mlp = WarmStartMLP(dev, seed=2)
    mlp.load_master(rng.standard_normal(M.N_PARAMS) * 0.15)
    X = rng.standard_normal((n, 16))
    X[:, 15] = 0
    Y = (rng.standard_normal((n, 4)) * 0.3).astype(np.float32)
    loss, grad = mlp.gradient(torch.as_tensor(X, dtype=torch.float32).to(torch.bfloat16).to(dev),
                              torch.as_tensor(Y).to(dev))
    ref_loss, ref = M.loss_and_grad(mlp.master.cpu().numpy(), M.bf16(X), Y, emulate=True)
    g = grad.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(g - ref) <= 5e-3 * np.linalg.norm(ref)
    assert abs(float(loss) - ref_loss) <= 5e-3 * ref_loss
