"""The Doppler least squares with a first row that says little or nothing: weight 0
or next to it, its Doppler far off.  Such a row must not cost the others their
digits.  Against the FP64 oracle; tolerances as in tests/test_doppler_sizes_gpu.py
(FP64 on both sides, log-weights stored in FP32; the tiny weight's own share of the
log-weight is of order one)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w0,off_hz", [(0.0, 1e6), (0.0, 1e12), (0.0, 1e200), (1e-12, 5e6), (1.0, 0.0)])
def test_first_row_of_no_weight(w0, off_hz):
    from gnss_gpu_b200 import ParticleFilterDevice
    rng = np.random.default_rng(4)
    n, m, wl = 300, 12, 0.19
    rx = np.array([-3957199.0, 3310205.0, 3737911.0])
    d = rng.normal(size=(m, 3))
    sat = rx + 2.1e7 * d / np.linalg.norm(d, axis=1, keepdims=True)
    sv, tv = rng.normal(0, 2000.0, (m, 3)), np.array([5.0, -3.0, 1.0])
    los = (sat - rx) / np.linalg.norm(sat - rx, axis=1, keepdims=True)
    dop = -(np.sum((sv - tv) * los, 1) + 300.0 + rng.normal(0, 0.2, m)) / wl
    w = rng.uniform(0.2, 2.0, m)
    w[0], dop[0] = w0, dop[0] + off_hz
    pf = ParticleFilterDevice(n_particles=n, sigma_pos=1.0, sigma_cb=1.0, seed=3, resampling="systematic")
    pf.initialize(rx, clock_bias=10.0, spread_pos=10.0, spread_cb=5.0, velocity=tv, spread_vel=1.0)
    st0 = pf.get_particle_states()
    pf.update_doppler(sat, sv, dop, velocity_update_gain=0.6, max_velocity_update_mps=1.5, weights=w, wavelength=wl,
                      sigma_mps=0.4, resample=False)
    use = w > 0.0
    lw, v, _ = O.doppler(st0[:, :3], st0[:, 4:7], st0[:, 7:], sat[use], sv[use], dop[use], w[use], wl, 0.4, gain=0.6,
                         max_update=1.5)
    st1 = pf.get_particle_states()
    np.testing.assert_allclose(st1[:, 4:7], v, rtol=1e-9, atol=1e-8)
    np.testing.assert_allclose(pf.get_log_weights(), lw, rtol=1e-6, atol=1e-6)
