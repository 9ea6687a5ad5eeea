"""Kepler's equation where ten Newton updates need not converge (eccentricities no
broadcast orbit has, which the call accepts): the position is still a point of the
orbit, its radius between perigee and apogee, and where plain Newton converges
without wandering it is the solution's.

Tolerances: the radius a (1 - e cos E) and the two rotations that follow carry a few
2^-53 each, and cos E of a rounded E at most 2^-53 more: 1e-12 of the apogee.  A
rounding of M (2^-52 pi) moves E by up to 1 / (1 - e) of it, 7e-13 at e = 0.999,
so positions agree within 2 a x 1e-12 x a few updates: 1e-3 m holds with room for
a hundred of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e", [0.9, 0.97, 0.98, 0.99, 0.999, 1.0 - 1e-9])
def test_position_stays_on_the_orbit(e):
    from gnss_gpu_b200 import _native as N
    from gnss_gpu_b200.ephemeris import broadcast_orbits
    ns = 4001
    M = np.linspace(-np.pi, np.pi, ns)
    rec = np.zeros(ns, N.BROADCAST_DTYPE)
    rec["system"] = ord("G")
    rec["kepler"]["sqrt_a"], rec["kepler"]["e"], rec["kepler"]["M0"] = 5153.7, e, M
    a = 5153.7 ** 2
    pos, clk = broadcast_orbits(rec, [0.0])
    r = np.linalg.norm(pos[0], axis=1)
    assert np.all(np.isfinite(pos)) and np.all(np.isfinite(clk))
    assert np.all(r <= a * (1.0 + e) * (1.0 + 1e-12)) and np.all(r >= a * (1.0 - e) - a * (1.0 + e) * 1e-12)
    E, far, dE = M.copy(), np.zeros(ns), np.ones(ns)
    for _ in range(10):
        dE = (M - E + e * np.sin(E)) / (1.0 - e * np.cos(E))
        E = E + dE
        far = np.maximum(far, np.abs(dE))
    ok = (np.abs(dE) < 1e-12) & (far < 1.0)
    assert ok.sum() > 1000
    want = np.stack([a * (np.cos(E) - e), a * np.sqrt(1.0 - e * e) * np.sin(E)], axis=1)
    np.testing.assert_allclose(pos[0][ok, :2], want[ok], rtol=0, atol=1e-3)


@pytest.mark.parametrize("e", [1.0, 1.2, 3.0])
def test_no_ellipse_leaves_the_clock_bounded(e):
    """The relativistic term is F e sqrt(A) sin E for some angle E, also where the
    equation has no solution the updates could find; at e = 1 and M = 0 the first
    update is 0 / 0, and the clock NaN."""
    from gnss_gpu_b200 import _native as N
    from gnss_gpu_b200.ephemeris import broadcast_orbits
    M = np.linspace(-np.pi, np.pi, 4001)
    rec = np.zeros(4001, N.BROADCAST_DTYPE)
    rec["system"] = ord("G")
    rec["kepler"]["sqrt_a"], rec["kepler"]["e"], rec["kepler"]["M0"] = 5153.7, e, M
    _, clk = broadcast_orbits(rec, [0.0])
    undefined = (M == 0.0) & (e == 1.0)
    assert undefined.sum() == (e == 1.0)
    np.testing.assert_array_equal(np.isnan(clk[0]), undefined)
    assert np.all(np.abs(clk[0][~undefined]) <= 4.442807633e-10 * e * 5153.7 * (1.0 + 1e-12))
