"""Observation terms at the edges of the kernel (one particle, remainders of a
block, 1 to 128 rows, reference satellites shared by none, some or all rows, gates
that keep fewer than three rows) against the FP64 oracle.  Tolerance: FP64 sums
on both sides (ranges of 2e7 m: 4e-9 m, 2e-8 cycles per residual, so a term w v dv /
sigma^2 of 128 rows stays below 1e-6 max(1, |lw|)) stored in FP32: 1e-6 relative;
particles with a residual within 1e-6 of the gate or of half a cycle are left out."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [O.OBS_DD_PSEUDORANGE, O.OBS_CARRIER_AFV, O.OBS_DD_CARRIER_AFV])
@pytest.mark.parametrize("n,rows,gate,hk,refs", [(1, 1, 0.0, 0.0, 1), (255, 2, 0.2, 0.0, 2), (256, 3, 0.2, 1.2, 1),
                                                 (257, 17, 0.2, 0.0, 3), (5000, 128, 0.3, 1.5, 128)])
def test_obs_term_matches_oracle_at_edges(kind, n, rows, gate, hk, refs):
    from gnss_gpu_b200 import _native as N
    from gnss_gpu_b200.engine import Engine, EngineOptions, FilterSpec
    rng = np.random.default_rng(n + rows + kind)
    p0 = np.array([-3957199.0, 3310205.0, 3737911.0])
    sky = lambda m: p0 + 2.1e7 * (lambda d: d / np.linalg.norm(d, axis=1, keepdims=True))(rng.normal(size=(m, 3)))  # noqa: E731
    dd = kind != O.OBS_CARRIER_AFV
    if not dd:
        gate = 0.0
    sk, ref = sky(rows), sky(refs)[np.sort(rng.integers(0, refs, rows))]
    wl = np.full(rows, 0.19) if kind != O.OBS_DD_PSEUDORANGE else np.ones(rows)
    bk, br = rng.uniform(2.0e7, 2.2e7, (2, rows))
    d = lambda s: np.linalg.norm(s - p0, axis=1)  # noqa: E731
    scale = 5.0 if kind == O.OBS_DD_PSEUDORANGE else 1.0
    obs = ((d(sk) - d(ref) - bk + br) if dd else d(sk) + 30.0) / wl + rng.normal(0, 0.15 * scale, rows)
    w = rng.uniform(0.5, 2.0, rows)
    r = np.zeros(rows, N.OBS_ROW_DTYPE)
    r["sat_k"], r["sat_ref"], r["obs"], r["base_k"], r["base_ref"], r["weight"], r["wavelength"] = sk, ref, obs, bk, br, w, wl
    eng = Engine([FilterSpec(n_particles=n, seed=3)], EngineOptions(n_clk=1, weight_mode="generic", max_sats=8))
    eng.initialize(0, p0, 30.0, 0.4 if kind else 2.0, 0.2)
    eng.add_obs_term(0, kind, r, 0.25 * scale, gate * scale, hk, accumulate=False)
    got = eng.state_f32(0)[1].astype(np.float64)
    x, _ = eng.state_f32(0)
    a, clk, _ = eng.anchor(0)
    rot, _ = eng.frame(0)
    want, res = O.obs_term(x, a, clk, rot, kind, sk, obs, w, ref, bk, br, wl, 0.25 * scale, gate * scale, hk)
    edge = np.zeros(n, bool)
    if gate > 0:
        edge |= np.any(np.abs(np.abs(res) - gate * scale) < 1e-6, axis=0)
    if kind != O.OBS_DD_PSEUDORANGE:
        edge |= np.any(np.abs(np.abs(res) - 0.5) < 1e-6, axis=0)
    assert edge.mean() < 0.01 or n == 1
    np.testing.assert_allclose(got[~edge], want[~edge], rtol=1e-6, atol=1e-6)
