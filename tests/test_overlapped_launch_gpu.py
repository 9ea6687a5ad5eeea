"""Calls whose kernels overlap their predecessor, one behind the other without a
wait on the host, against the same calls with a wait after each: the same bytes.
(Training steps on the same parameters; orbits whose GLONASS table comes to the
same scratch memory with other records each time.)"""
import numpy as np
import pytest

from gnss_gpu_b200 import _native as N
from oracle import mlp_oracle as M
from test_mlp_gpu import _data, _dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 3000, 20_000])
def test_training_steps_back_to_back(n):
    import torch
    L = N.load()
    X, Y = _data(n, n)
    dx, dy = _dev(X, torch), _dev(Y, torch)
    scratch = torch.zeros(L.pf_mlp_scratch_bytes(), dtype=torch.uint8, device="cuda")

    def train(wait):
        p, m, v = _dev(M.init_params(3), torch), *(torch.zeros(M.N_PARAMS, device="cuda") for _ in range(2))
        loss = torch.zeros(40, device="cuda")
        torch.cuda.synchronize()
        for k in range(40):
            N.check(L.pf_mlp_adam_step(dx.data_ptr(), dy.data_ptr(), n, p.data_ptr(), m.data_ptr(), v.data_ptr(),
                                       k + 1, 1e-2, loss[k:].data_ptr(), scratch.data_ptr(), scratch.numel(), None))
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return [t.cpu().numpy() for t in (p, m, v, loss)]

    want = train(True)
    for _ in range(3):
        for g, w in zip(train(False), want):
            np.testing.assert_array_equal(g, w)


def test_glonass_orbits_back_to_back():
    import torch
    L = N.load()
    rng = np.random.default_rng(2)
    ne, ns, calls = 2000, 24, 6
    t = torch.arange(ne, dtype=torch.float64, device="cuda") * 3.0
    recs = []
    for _ in range(calls):
        rec = np.zeros(ns, N.BROADCAST_DTYPE)
        rec["system"] = ord("R")
        g, a = rec["glonass"], rng.uniform(0, 2 * np.pi, ns)
        vel = np.sqrt(3.9860044e14 / 2.55e7)
        g["toe"] = rng.uniform(0, 6000, ns)
        g["pos"] = 2.55e7 * np.stack([np.cos(a), np.sin(a), 0 * a], 1)
        g["vel"] = vel * np.stack([-0.43 * np.sin(a), 0.43 * np.cos(a), 0.9 + 0 * a], 1)
        recs.append(torch.from_numpy(rec.view(np.uint8).copy()).cuda())

    def run(wait):
        pos = torch.zeros((calls, ne, ns, 3), dtype=torch.float64, device="cuda")
        clk = torch.zeros((calls, ne, ns), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        for c in range(calls):
            N.check(L.pf_broadcast_orbits(recs[c].data_ptr(), ns, None, t.data_ptr(), ne, ns, 60.0, pos[c].data_ptr(),
                                          clk[c].data_ptr(), None))
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return pos.cpu().numpy(), clk.cpu().numpy()

    want = run(True)
    assert np.isfinite(want[0]).all() and len(np.unique(want[0][:, 100, 0, 0])) == calls
    for _ in range(3):
        got = run(False)
        np.testing.assert_array_equal(got[0], want[0])
        np.testing.assert_array_equal(got[1], want[1])
