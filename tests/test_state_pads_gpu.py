"""Slots past a filter's last particle, up to the next multiple of four: the state
is read in groups of four, so every writer of a state buffer leaves them finite,
whatever the workspace held before.  The engine gets memory filled with 0xFF bytes
(NaN); particle counts of every remainder go through the velocity predict (its
output buffer is one that nothing has written yet), with and without a pending
resample, and through a checkpoint restored into the second state buffer.

Tolerances: velocities and covariances are FP64 on both sides (1e-12); positions
are FP32 offsets about an anchor within 50 m, rounded once per predict and once per
recentring (2e-5 m); the estimate is the weighted mean of the same particles from
FP32 sums (1 mm)."""
import gc

import numpy as np
import pytest

from gnss_gpu_b200 import _native as N
from oracle import oracle as O

import pfhelp as H
from conftest import TOKYO_PR, TOKYO_SATS, TOKYO_TRUE_CB, TOKYO_TRUE_POS

pytestmark = pytest.mark.gpu


def _on_poisoned_memory(make, engine):
    """make() again, its engine's workspace on memory filled with 0xFF."""
    import torch
    first = make()
    nbytes = engine(first).workspace.numel()
    del first
    gc.collect()
    bad = torch.full((nbytes,), 0xFF, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    at = bad.data_ptr()
    del bad
    got = make()
    assert engine(got).workspace.data_ptr() == at
    return got


def _mean(states, log_w):
    w = np.exp(log_w - log_w.max())
    return (states[:, :4] * w[:, None]).sum(0) / w.sum()


@pytest.mark.parametrize("kf", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 255, 257, 1001])
def test_velocity_predict_at_every_remainder(n, kf):
    from gnss_gpu_b200 import ParticleFilterDevice

    def make():
        pf = ParticleFilterDevice(n_particles=n, seed=77, resampling="systematic", sigma_vel=0.0 if kf else 0.7,
                                  velocity_guide_alpha=0.6, rbpf_velocity_kf=kf, velocity_process_noise=0.3,
                                  ess_threshold=1.0)
        pf.initialize(TOKYO_TRUE_POS, clock_bias=TOKYO_TRUE_CB, spread_pos=5.0, spread_cb=3.0,
                      velocity=np.array([3.0, -1.0, 0.5]), spread_vel=1.5, velocity_init_sigma=0.8)
        return pf

    pf = _on_poisoned_memory(make, lambda p: p._engine)
    guide = np.array([2.0, 1.0, -0.5])

    def predict_and_check(before):
        pf.predict(velocity=guide, dt=0.5, sigma_pos=0.4)
        want = O.vel_predict(before[:, :3], before[:, 4:7], before[:, 7:], guide, 0.5, 0.4, 0.0 if kf else 0.7, 0.6,
                             kf, 0.3, pf._step, 77)
        pf._flush()
        est = pf.estimate()
        got = pf.get_particle_states()
        np.testing.assert_allclose(got[:, :3], want[0], rtol=0, atol=2e-5)
        np.testing.assert_allclose(got[:, 4:7], want[1], rtol=1e-12, atol=1e-12)
        np.testing.assert_allclose(got[:, 7:], want[2], rtol=1e-12, atol=1e-12)
        np.testing.assert_allclose(est, _mean(got, np.asarray(pf.get_log_weights())), rtol=0, atol=1e-3)
        return got

    st = predict_and_check(pf.get_particle_states())       # into the buffer nothing has written yet
    pf.update(TOKYO_SATS, TOKYO_PR, None, resample=False)  # and from it
    np.testing.assert_allclose(pf.estimate(), _mean(st, np.asarray(pf.get_log_weights())), rtol=0, atol=1e-3)
    st = pf.get_particle_states()
    pf.update(TOKYO_SATS, TOKYO_PR, None, resample=True)
    anc = pf.get_resample_ancestors() if n > 1 else np.zeros(1, int)
    if n > 1:
        assert len(np.unique(anc)) < n
    predict_and_check(st[anc])                             # through the pending resample
    pf.update(TOKYO_SATS, TOKYO_PR, None, resample=False)
    st = pf.get_particle_states()
    assert np.all(np.isfinite(st))
    np.testing.assert_allclose(pf.estimate(), _mean(st, np.asarray(pf.get_log_weights())), rtol=0, atol=1e-3)


@pytest.mark.parametrize("n", [5, 6, 7, 1001])
def test_checkpoint_restored_into_the_second_buffer(n):
    def make():
        eng = H.make_engine([n], seeds=[11], ess=0.0)
        eng.initialize(0, TOKYO_TRUE_POS, TOKYO_TRUE_CB, 5.0, 3.0)
        return eng

    fl = N.PF_EP_PREDICT | N.PF_EP_WEIGHT
    a = make()
    fe, sv = a.pack_epoch([dict(sats=TOKYO_SATS, pr=TOKYO_PR, flags=fl | N.PF_EP_FORCE_RESAMPLE)])
    a.step_io(fe, sv)
    fe, sv = a.pack_epoch([dict(sats=TOKYO_SATS, pr=TOKYO_PR, flags=fl | N.PF_EP_NO_RESAMPLE)])
    a.step_io(fe, sv)
    a.step_io(fe, sv)          # three steps: the second buffer is current, no gather pending
    blob = a.checkpoint(0)
    a.step_io(fe, sv)
    want = a.results()[0]
    del a
    b = _on_poisoned_memory(make, lambda e: e)
    b.restore(0, blob)
    b.step_io(fe, sv)
    got = b.results()[0]
    for key in ("est_ecef", "est_clk", "cov_enu", "ess"):
        np.testing.assert_array_equal(got[key], want[key])
