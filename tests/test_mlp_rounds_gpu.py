"""Gradient and Adam step at the edges of the training kernel's rounds (64 rows
per CTA, 296 CTAs, remainders of a 16-row warp tile).  The gradient's tolerance
is that of tests/test_mlp_gpu.py (BF16 operands, FP32 sums in another order); an
Adam step moves a parameter by lr g / (|g| + eps), compared where |g| is above 5 %
of the largest, with the gradient's 2 % in both numerator and denominator: the step
is lr times a value within 1e-6 of +-1 there."""
import numpy as np
import pytest

from gnss_gpu_b200 import _native as N
from oracle import mlp_oracle as M
from test_mlp_gpu import _data, _dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [15, 16, 17, 63, 64, 65, 18_944, 18_945, 37_950])
def test_gradient_and_step_at_round_edges(n):
    import torch
    L = N.load()
    X, Y = _data(n, n)
    prm = M.init_params(3)
    dx, dy, dp = _dev(X, torch), _dev(Y, torch), _dev(prm, torch)
    grad, m, v = (torch.zeros(M.N_PARAMS, device="cuda") for _ in range(3))
    loss = torch.zeros(1, device="cuda")
    scratch = torch.zeros(L.pf_mlp_scratch_bytes(), dtype=torch.uint8, device="cuda")
    N.check(L.pf_mlp_grad(dx.data_ptr(), dy.data_ptr(), n, dp.data_ptr(), grad.data_ptr(), loss.data_ptr(),
                          scratch.data_ptr(), scratch.numel(), None))
    N.check(L.pf_mlp_adam_step(dx.data_ptr(), dy.data_ptr(), n, dp.data_ptr(), m.data_ptr(), v.data_ptr(), 1, 1e-2,
                               loss.data_ptr(), scratch.data_ptr(), scratch.numel(), None))
    torch.cuda.synchronize()
    lo, go = M.loss_grad(prm, X, Y, bf=True)
    g = grad.cpu().numpy().astype(np.float64)
    assert float(loss.item()) == pytest.approx(lo, rel=2e-3)
    scale = np.abs(go).max()
    assert np.max(np.abs(g - go)) <= 2e-2 * scale and np.mean(np.abs(g - go)) <= 1e-3 * scale
    big = np.abs(go) > 0.05 * scale
    step = (dp.cpu().numpy() - np.asarray(prm, np.float32))[big]
    np.testing.assert_allclose(step, -1e-2 * np.sign(go[big]), atol=1e-2 * 1e-3)
