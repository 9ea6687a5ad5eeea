"""Broadcast orbits at the edges of the kernel's tiles and of its shortened
angle arithmetic, against the FP64 oracle: odd epoch and satellite counts (both
tile shapes), missing records, eccentric orbits, correction angles on both sides
of the small-angle limit, whole and fractional GLONASS step lengths.

Tolerance: an ECEF coordinate is a product of a ~2.7e7 m radius and angles of up
to ~20 rad, each within a few 2^-53, times 1 / (1 - e) <= 5 for the anomaly:
2.7e7 x 20 x 4 x 1.1e-16 x 5 = 1.2e-6 m; clocks within 1e-15 s."""
import numpy as np
import pytest

from oracle import orbit as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne,ns,step", [(1, 1, 60.0), (31, 9, 60.0), (33, 8, 59.3), (130, 17, 60.0), (9000, 67, 60.0)])
def test_orbits_match_oracle_at_tile_edges(ne, ns, step):
    from gnss_gpu_b200 import _native as N
    from gnss_gpu_b200.ephemeris import broadcast_orbits
    rng = np.random.default_rng(ne + ns)
    nr = 2 * ns
    rec = np.zeros(nr, N.BROADCAST_DTYPE)
    kind = rng.choice(list("GEJCR"), nr)
    rec["system"] = [ord(c) for c in kind]
    for r in range(nr):
        if kind[r] == "R":
            g = rec["glonass"][r:r + 1]
            a, v = rng.uniform(0, 6.28), np.sqrt(3.9860044e14 / 2.55e7)
            g["toe"], g["tau_n"], g["gamma_n"] = rng.uniform(0, 6000), 1e-5, 1e-12
            g["pos"] = (2.55e7 * np.cos(a), 2.55e7 * np.sin(a), 0.0)
            g["vel"] = (-0.43 * v * np.sin(a), 0.43 * v * np.cos(a), 0.9 * v)
            g["acc"] = rng.uniform(-3e-6, 3e-6, 3)
            continue
        k = rec["kepler"][r:r + 1]
        k["sqrt_a"], k["e"] = rng.uniform(5100, 5450), rng.choice([0.0, 0.001, 0.02, 0.3, 0.8])
        for f in ("i0", "omega0", "omega", "M0"):
            k[f] = rng.uniform(-3, 3)
        k["delta_n"], k["omega_dot"], k["idot"] = 4.5e-9, -8e-9, rng.choice([0.0, 5e-10, 2e-5])
        big = rng.choice([1e-6, 0.02, 0.2])
        for f in ("cuc", "cus", "cic", "cis"):
            k[f] = rng.uniform(-big, big)
        k["crc"], k["crs"] = 220.0, -14.0
        k["toe"] = k["toc"] = rng.uniform(0, 6000)
        k["af0"], k["af1"], k["tgd"] = 1e-4, -1e-12, 1e-8
    t = np.sort(rng.uniform(0.0, 6000.0, ne))
    idx = rng.integers(0, 2, (ne, ns)).astype(np.int32) * ns + np.arange(ns, dtype=np.int32)
    idx[rng.random((ne, ns)) < 0.05] = -1
    pos, clk = broadcast_orbits(rec, t, idx, glo_step=step)
    es, ss = np.nonzero(idx >= 0)
    assert np.isnan(pos[idx < 0]).all() and np.isnan(clk[idx < 0]).all()
    pick = rng.choice(len(es), min(len(es), 400), replace=False)
    for e, s in zip(es[pick], ss[pick]):
        r = idx[e, s]
        if kind[r] == "R":
            g = rec["glonass"][r]
            st = {"toe": float(g["toe"]), "pos": g["pos"], "vel": g["vel"], "acc": g["acc"], "tau_n": float(g["tau_n"]),
                  "gamma_n": float(g["gamma_n"])}
            p, c = O.glonass(st, float(t[e]), step)
        else:
            p, c = O.kepler({f: float(rec["kepler"][f][r]) for f in N.EPHEMERIS_FIELDS}, kind[r], [t[e]])
            p, c = p[0], c[0]
        np.testing.assert_allclose(pos[e, s], p, rtol=0, atol=1.2e-6)
        assert abs(clk[e, s] - c) <= 1e-15
