"""The MLP training kernel's swizzled tiles and split partial sums: gradients against the numpy oracle at row counts around
the 128-row CTA and the eight-way split of the partials, and packed weights off a 16-byte boundary against aligned ones
(the same bits).  The gradient's tolerance is the one of the BF16-emulating oracle comparison (5e-3 relative L2)."""
import ctypes as C

import numpy as np
import pytest

from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


def _setup(n, seed=1):
    import torch
    from diffphd_b200.warmstart import WarmStartMLP
    dev = torch.device("cuda:0")
    mlp = WarmStartMLP(dev, seed=seed)
    rng = np.random.default_rng(seed)
    mlp.load_master(rng.standard_normal(M.N_PARAMS) * 0.15)
    X = rng.standard_normal((n, 16))
    X[:, 15] = 0
    Y = rng.standard_normal((n, 4)) * 0.3
    return (mlp, torch.as_tensor(X, dtype=torch.float32).to(torch.bfloat16).to(dev),
            torch.as_tensor(Y, dtype=torch.float32).to(dev), M.bf16(X), Y.astype(np.float32))


@pytest.mark.parametrize("n", [1, 127, 129, 128 * 7, 128 * 9 + 5, 128 * 20])
def test_gradient_at_partial_counts(n):
    mlp, Xb, Yb, X, Y = _setup(n)
    loss, grad = mlp.gradient(Xb, Yb)
    ref_loss, ref = M.loss_and_grad(mlp.master.cpu().numpy(), X, Y, emulate=True)
    g = grad.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(g - ref) <= 5e-3 * np.linalg.norm(ref)
    assert abs(float(loss) - ref_loss) <= 5e-3 * ref_loss


def test_packed_weights_off_a_16_byte_boundary():
    import torch
    from diffphd_b200 import core
    mlp, Xb, Yb, _, _ = _setup(300)
    L, p = core.load_library(), lambda t: C.c_void_p(t.data_ptr())
    shifted = torch.zeros(mlp.n_packed + 8, dtype=torch.bfloat16, device=Xb.device)
    outs = []
    for packed in (mlp.packed, shifted[1:1 + mlp.n_packed]):
        packed.copy_(mlp.packed)
        out = torch.zeros(300, 8, device=Xb.device)
        core.Deformable._check(L.dphd_mlp_forward(p(mlp.master), p(packed), p(Xb), 300, p(out), None))
        grad = torch.zeros_like(mlp.master)
        core.Deformable._check(L.dphd_mlp_train_step(
            p(mlp.master), p(packed), p(Xb), p(Yb), 300, p(mlp._partials(300)), 0.0, 0.9, 0.999, 1e-8, 0.0, 1,
            p(mlp.m), p(mlp.v), p(grad), p(mlp.loss_buf), None))
        torch.cuda.synchronize()
        outs.append((out, grad))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
