"""The 3D likelihood's three ways to its rays (a thread per ray, per particle,
shadow cells) against one ray per (particle, satellite) of the line-of-sight
query, with the likelihood's formula in FP64.

Tolerance: the log-weight is an FP32 rounding of an FP64 sum, |d lw| <= 1e-5
max(1, |lw|); the flags may differ where a ray grazes an edge (the query forms
its origin from exported particles, one rounding apart): at most 2 rays in
100,000, and at least one satellite both blocked and clear."""
import ctypes as C

import numpy as np
import pytest

from test_bvh_host import city_mesh

pytestmark = pytest.mark.gpu

S_LOS, S_NLOS, BIAS = 3.0, 30.0, 20.0


@pytest.mark.parametrize("n,n_sat,spread,fail", [
    (1, 1, 1.0, False), (33, 5, 30.0, False), (31_251, 32, 10.0, False),          # thread per ray, up to its limit
    (31_253, 32, 10.0, False), (2_000, 24, 10.0, True),                            # thread per particle, and without scratch
    (34_376, 64, 3.0, False), (220_003, 11, 0.02, False), (300_001, 17, 25.0, False),  # cells: 64 satellites, a point cloud, a wide one
])
def test_rays_equal_line_of_sight_query(n, n_sat, spread, fail):
    from gnss_gpu_b200 import BVHAccelerator
    from gnss_gpu_b200 import _native as N
    from gnss_gpu_b200.engine import Engine, EngineOptions, FilterSpec
    rng = np.random.default_rng(3)
    tri, anchor, rot, _ = city_mesh(5, 800.0)
    bvh = BVHAccelerator(tri)
    az, el = rng.uniform(0, 2 * np.pi, n_sat), rng.uniform(np.radians(8), np.radians(70), n_sat)
    start = anchor + np.array([400.0, 400.0, 1.5]) @ rot
    sats = start + 2.2e7 * (np.stack([np.cos(el) * np.sin(az), np.cos(el) * np.cos(az), np.sin(el)], 1) @ rot)
    pr = np.linalg.norm(sats - start, axis=1) + 50.0 + rng.normal(0, 10.0, n_sat)
    w = rng.uniform(0.3, 1.0, n_sat)
    eng = Engine([FilterSpec(n_particles=n, seed=5)], EngineOptions(n_clk=1, max_sats=64))
    eng.initialize(0, start, 50.0, spread, 5.0)
    if n > 1000:  # a few particles far outside any grid of the cloud
        st, lw = eng.state_f32(0)
        st[:3, ::997] *= 9.0
        eng.set_state_f32(0, st, lw)
    if fail:
        N.check(N.load().pf_test_fail_alloc(1))
    eng.add_3d_term(0, bvh.mesh, sats, pr, w, S_LOS, S_NLOS, BIAS, 1.0, 0.0)
    N.check(N.load().pf_test_fail_alloc(0))
    p = eng.particles(0)
    got = eng.state_f32(0)[1].astype(np.float64)
    clear = np.concatenate([bvh.check_los_batch(q[:, :3], np.broadcast_to(sats, (len(q), n_sat, 3)))
                            for q in np.array_split(p, max(1, n // 50_000))])
    r = pr - (np.linalg.norm(sats - p[:, None, :3], axis=2) + p[:, 3:4])
    los = -0.5 * w * r * r / S_LOS ** 2
    rn = np.where(r > 0, r - BIAS, r)
    want = np.where(clear, los, -0.5 * w * rn * rn / S_NLOS ** 2).sum(1)
    off = np.abs(got - want) > 1e-5 * np.maximum(1.0, np.abs(want))
    assert off.sum() <= np.ceil(2e-5 * n * n_sat) if n > 1000 else not off.any()
    if n > 1000 and spread >= 3.0:
        share = clear.mean(0)
        assert np.any((share > 0.001) & (share < 0.999))
