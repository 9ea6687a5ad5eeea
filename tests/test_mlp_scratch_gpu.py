"""Gradient and Adam step with less scratch than pf_mlp_scratch_bytes(): from 64
partial gradients up (what a caller that sized its scratch once may hold) the calls
run, on fewer CTAs; below they are refused.  The gradient's tolerance is that of
tests/test_mlp_gpu.py; an Adam step's that of tests/test_mlp_rounds_gpu.py.  Bytes
behind the scratch stay as they were."""
import numpy as np
import pytest

from gnss_gpu_b200 import _native as N
from oracle import mlp_oracle as M
from test_mlp_gpu import _data, _dev

pytestmark = pytest.mark.gpu

ROW = (M.N_PARAMS + 1) * 4


@pytest.mark.parametrize("rows,n", [(64, 5000), (64, 40_001), (100, 40_001), (295, 40_001)])
def test_smaller_scratch_is_enough(rows, n):
    import torch
    L = N.load()
    X, Y = _data(n, n)
    prm = M.init_params(3)
    dx, dy, dp = _dev(X, torch), _dev(Y, torch), _dev(prm, torch)
    grad, m, v = (torch.zeros(M.N_PARAMS, device="cuda") for _ in range(3))
    loss = torch.zeros(1, device="cuda")
    scratch = torch.full((rows * ROW + 4096,), 0x5A, dtype=torch.uint8, device="cuda")
    N.check(L.pf_mlp_grad(dx.data_ptr(), dy.data_ptr(), n, dp.data_ptr(), grad.data_ptr(), loss.data_ptr(),
                          scratch.data_ptr(), rows * ROW, None))
    N.check(L.pf_mlp_adam_step(dx.data_ptr(), dy.data_ptr(), n, dp.data_ptr(), m.data_ptr(), v.data_ptr(), 1, 1e-2,
                               loss.data_ptr(), scratch.data_ptr(), rows * ROW, None))
    torch.cuda.synchronize()
    assert bool((scratch[rows * ROW:] == 0x5A).all())
    lo, go = M.loss_grad(prm, X, Y, bf=True)
    g = grad.cpu().numpy().astype(np.float64)
    assert float(loss.item()) == pytest.approx(lo, rel=2e-3)
    scale = np.abs(go).max()
    assert np.max(np.abs(g - go)) <= 2e-2 * scale and np.mean(np.abs(g - go)) <= 1e-3 * scale
    big = np.abs(go) > 0.05 * scale
    step = (dp.cpu().numpy() - np.asarray(prm, np.float32))[big]
    np.testing.assert_allclose(step, -1e-2 * np.sign(go[big]), atol=1e-2 * 1e-3)


def test_too_little_scratch_is_refused():
    import torch
    L = N.load()
    t = torch.zeros(M.N_PARAMS, device="cuda")
    s = torch.zeros(64 * ROW, dtype=torch.uint8, device="cuda")
    assert L.pf_mlp_grad(t.data_ptr(), t.data_ptr(), 8, t.data_ptr(), t.data_ptr(), None, s.data_ptr(),
                         64 * ROW - 1, None) == N.PF_EINVAL
