"""Doppler terms at the edges of the kernel (one particle, remainders of a
block, 1 to 64 rows, zero weights, asymmetric and zero covariances) against the
FP64 oracle.  With fewer than four weighted rows the least-squares system is
singular but for its 1e-9 diagonal, and one rounding of a line of sight moves the
undetermined part of the velocity by 1e-16 / 1e-9 (the oracle is then 4e-8 off
60-digit arithmetic itself), so there only the log-weights are compared.  Tolerance: both sides are FP64 over the same formulas in another
order; the 4x4 normal equations have condition numbers up to about 1e4 here
(clustered skies), so velocities agree to 1e-9 relative with room for 1e4 x
1e-13, log-weights to the FP32 they are stored in."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kf", [False, True])
@pytest.mark.parametrize("n,m", [(1, 1), (1, 64), (127, 3), (128, 4), (129, 5), (1000, 64), (257, 20)])
def test_doppler_matches_oracle_at_edges(n, m, kf):
    from gnss_gpu_b200 import ParticleFilterDevice
    rng = np.random.default_rng(n + 7 * m)
    rx = np.array([-3957199.0, 3310205.0, 3737911.0])
    d = rng.normal(size=(m, 3))
    sat = rx + 2.1e7 * d / np.linalg.norm(d, axis=1, keepdims=True)
    sv = rng.normal(0, 2000.0, (m, 3))
    tv, wl = np.array([5.0, -3.0, 1.0]), 0.19
    los = (sat - rx) / np.linalg.norm(sat - rx, axis=1, keepdims=True)
    dop = -(np.sum((sv - tv) * los, 1) + 300.0 + rng.normal(0, 0.2, m)) / wl
    w = rng.uniform(0.2, 2.0, m)
    w[1::5] = 0.0
    pf = ParticleFilterDevice(n_particles=n, sigma_pos=1.0, sigma_cb=1.0, seed=3, resampling="systematic")
    pf.initialize(rx, clock_bias=10.0, spread_pos=10.0, spread_cb=5.0, velocity=tv, spread_vel=1.0)
    st = np.zeros((n, 16))
    st[:, :4] = pf.get_particles()
    st[:, 4:7] = tv + rng.normal(0, 2.0, (n, 3))
    a = rng.normal(0, 1.0, (n, 3, 3))
    P = a @ a.transpose(0, 2, 1)
    P[::3] += rng.normal(0, 0.05, (len(P[::3]), 3, 3))   # asymmetric
    P[1::7] = 0.0
    st[:, 7:] = P.reshape(n, 9)
    pf.set_particle_states(st)
    st0 = pf.get_particle_states()
    kw = dict(weights=w, wavelength=wl, sigma_mps=0.4, resample=False)
    if kf:
        pf.update_doppler_kf(sat, sv, dop, **kw)
    else:
        pf.update_doppler(sat, sv, dop, velocity_update_gain=0.6, max_velocity_update_mps=1.5, **kw)
    lw, v, Pw = O.doppler(st0[:, :3], st0[:, 4:7], st0[:, 7:], sat, sv, dop, w, wl, 0.4, gain=0.6, max_update=1.5,
                          kf=kf)
    st1 = pf.get_particle_states()
    if kf or m < 4 or np.sum(w > 0) >= 4:
        np.testing.assert_allclose(st1[:, 4:7], v, rtol=1e-9, atol=1e-8)
    np.testing.assert_allclose(st1[:, 7:], Pw.reshape(n, 9), rtol=1e-9, atol=1e-9)
    np.testing.assert_allclose(pf.get_log_weights(), lw, rtol=1e-6, atol=1e-6)
