"""Clouds too wide for shadow cells: their rays walk the hierarchy one by one, with
the verdicts of the line-of-sight query (the check and its tolerance are those of
tests/test_pf3d_rays_gpu.py), and in about the time of a call that has no scratch
for cells at all.  The cells took twice that time on such clouds; a third is left for
the grid that is tried first and for the clocks."""
import time

import numpy as np
import pytest

from test_bvh_host import city_mesh
from test_pf3d_rays_gpu import test_rays_equal_line_of_sight_query as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_sat,spread", [(150_001, 16, 90.0), (150_001, 16, 400.0), (34_377, 64, 150.0)])
def test_wide_clouds_equal_line_of_sight_query(n, n_sat, spread):
    _check(n, n_sat, spread, False)


def test_wide_cloud_costs_no_more_than_its_walks():
    from gnss_gpu_b200 import BVHAccelerator
    from gnss_gpu_b200 import _native as N
    from gnss_gpu_b200.engine import Engine, EngineOptions, FilterSpec
    rng = np.random.default_rng(3)
    tri, anchor, rot, _ = city_mesh(9, 2000.0)
    bvh = BVHAccelerator(tri)
    start = anchor + np.array([1000.0, 1000.0, 1.5]) @ rot
    az, el = rng.uniform(0, 2 * np.pi, 16), rng.uniform(0.15, 1.2, 16)
    sats = start + 2.2e7 * (np.stack([np.cos(el) * np.sin(az), np.cos(el) * np.cos(az), np.sin(el)], 1) @ rot)
    pr = np.linalg.norm(sats - start, axis=1) + 50.0
    eng = Engine([FilterSpec(n_particles=500_000, seed=5)], EngineOptions(n_clk=1, max_sats=64))
    eng.initialize(0, start, 50.0, 300.0, 5.0)

    def call(walk):
        if walk:
            N.check(N.load().pf_test_fail_alloc(1))
        t = time.perf_counter()
        eng.add_3d_term(0, bvh.mesh, sats, pr, np.ones(16), 3.0, 30.0, 20.0, 0.9, 0.05)
        dt = time.perf_counter() - t
        N.check(N.load().pf_test_fail_alloc(0))
        return dt

    times = np.array([[call(True), call(False)] for _ in range(15)])[3:]
    walk, here = np.median(times, axis=0)
    assert here < 1.33 * walk
