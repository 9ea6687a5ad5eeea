"""The performance cases of the particle-filter framework.

A case is one pass of work that a program built on this package has the GPU
do: an epoch of one filter, of a fleet, of the device filter with its
observation terms, of a building-aware filter, the orbits that feed them, a
training step of the NLOS network.  `listed()` names the cases, `draw()` gives
more of the same ranges, `prepare()` makes what the program holds before the
call, `run()` is one pass, `work()` its bytes and operations, `exact()` what
the pass returns in 64-bit arithmetic, written without the package.

Receivers drive a closed circle of RING epochs, so a filter can be stepped
for as long as wanted with the same inputs and stay converged.  Statistics
that the kernels form from FP32 sums (covariance, ESS, clock estimates) are
returned as FP32.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch

RING = 8                # epochs of a drive
LAT, LON, ALT = 35.63, 139.78, 40.0
WGS_A, WGS_F = 6378137.0, 1.0 / 298.257223563
ORBIT = 26_560_000.0    # radius of the satellites, m
SIGMA_PR = 5.0
WL = 0.19029367279836488


# ------------------------------------------------------------------- cases
def listed():
    return [
        # a receiver's own filter: a few thousand particles, GPS only, one
        # call per epoch from host records to host results (latency)
        dict(name="live-2k", kind="step", filters=1, n=2_000, n_max=2_000, sats=8, sats_min=8, clocks=1,
             resampler="systematic", iters=15, weight="gaussian"),
        # the benchmark's filter: 1M particles, four constellations with a
        # clock each
        dict(name="step-1m", kind="step", filters=1, n=1_000_000, n_max=1_000_000, sats=32, sats_min=32, clocks=4,
             resampler="systematic", iters=15, weight="gaussian"),
        # the same with the Megopolis resampler, the reference's default
        dict(name="megopolis-1m", kind="step", filters=1, n=1_000_000, n_max=1_000_000, sats=32, sats_min=32,
             clocks=4, resampler="megopolis", iters=32, weight="gaussian"),
        # a server's fleet: 256 independent receivers of uneven size, robust
        # (Huber) likelihood, satellite counts changing every epoch
        dict(name="fleet-256", kind="step", filters=256, n=1_000, n_max=100_000, sats=40, sats_min=6, clocks=1,
             resampler="systematic", iters=15, weight="huber"),
        # a fleet with the learned NLOS likelihood (network and mixture in
        # the epoch kernel)
        dict(name="learned-64", kind="step", filters=64, n=100_000, n_max=100_000, sats=24, sats_min=24, clocks=1,
             resampler="systematic", iters=15, weight="mixture"),
        # the reference's device filter with its robust options, defaults
        # otherwise (Megopolis, 15 iterations)
        dict(name="device-robust-1m", kind="device", n=1_000_000, sats=10, likelihood="student_t", gate=True,
             resampling="megopolis"),
        # differenced pseudoranges, then differenced carrier phase, gated and
        # with the Huber cost: the centimetre epoch of the device filter
        dict(name="dd-carrier-200k", kind="dd", n=200_003, pairs=14, gate=True, huber=True),
        # Rao-Blackwellised velocities: covariance-shaped predict, weights,
        # Doppler Kalman update per particle
        dict(name="doppler-kf-300k", kind="doppler", n=300_001, sats=11, kf=True),
        # sampled velocities: predict with velocity noise, weights, Doppler
        # likelihood and least-squares blend per particle
        dict(name="doppler-blend-1m", kind="doppler", n=1_000_000, sats=16, kf=False),
        # a building-aware filter in a 2 km city of about 10,000 triangles, a
        # ray per particle and satellite
        dict(name="city-1m", kind="city", n=1_000_000, sats=16, cell=40.0, spread=20.0),
        # input formation: a day at 1 Hz of 64 satellites, 40 of them Kepler
        # records and 24 GLONASS states
        dict(name="orbits-day", kind="orbits", epochs=86_400, kepler=40, glonass=24),
        # a training step of the NLOS network on its default batch
        dict(name="train-8192", kind="train", rows=8_192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "fleet", "device", "dd", "doppler", "city", "orbits", "train"])
    if kind == "step":
        n = _log_int(rng, 1_000, 2_000_000)
        clocks = rng.choice([1, 1, 2, 4])
        s = rng.randint(max(5, 2 * clocks), 40)
        return dict(kind="step", filters=1, n=n, n_max=n, sats=s, sats_min=s, clocks=clocks,
                    resampler=rng.choice(["systematic", "megopolis"]), iters=rng.choice([15, 32]),
                    weight=rng.choice(["gaussian", "gaussian", "huber"]))
    if kind == "fleet":
        lo = _log_int(rng, 500, 20_000)
        return dict(kind="step", filters=_log_int(rng, 4, 256), n=lo, n_max=lo * rng.randint(1, 4),
                    sats=rng.randint(20, 40), sats_min=rng.randint(6, 20), clocks=1, resampler="systematic", iters=15,
                    weight=rng.choice(["gaussian", "huber", "mixture"]))
    if kind == "device":
        return dict(kind="device", n=_log_int(rng, 10_000, 1_000_000), sats=rng.randint(6, 24),
                    likelihood=rng.choice(["gaussian", "student_t", "huber", "gmm"]), gate=rng.random() < 0.5,
                    resampling=rng.choice(["megopolis", "systematic"]))
    if kind == "dd":
        return dict(kind="dd", n=_log_int(rng, 10_000, 1_000_000), pairs=rng.randint(4, 24), gate=rng.random() < 0.5,
                    huber=rng.random() < 0.5)
    if kind == "doppler":
        return dict(kind="doppler", n=_log_int(rng, 10_000, 1_000_000), sats=rng.randint(5, 20),
                    kf=rng.random() < 0.5)
    if kind == "city":
        return dict(kind="city", n=_log_int(rng, 10_000, 1_000_000), sats=rng.randint(5, 24),
                    cell=rng.choice([40.0, 80.0]), spread=round(rng.uniform(3.0, 40.0), 1))
    if kind == "orbits":
        return dict(kind="orbits", epochs=_log_int(rng, 60, 86_400), kepler=rng.randint(8, 40),
                    glonass=rng.randint(0, 24))
    return dict(kind="train", rows=_log_int(rng, 500, 100_000))


# ---------------------------------------------------------------- geometry
def _frame():
    """ECEF point of the drives and its ECEF -> E/N/U rotation."""
    la, lo = math.radians(LAT), math.radians(LON)
    sl, cl, so, co = math.sin(la), math.cos(la), math.sin(lo), math.cos(lo)
    e2 = WGS_F * (2.0 - WGS_F)
    nn = WGS_A / math.sqrt(1.0 - e2 * sl * sl)
    p = np.array([(nn + ALT) * cl * co, (nn + ALT) * cl * so, (nn * (1.0 - e2) + ALT) * sl])
    rot = np.array([[-so, co, 0.0], [-sl * co, -sl * so, cl], [cl * co, cl * so, sl]])
    return p, rot


def _sky(rng, p, rot, n):
    """n satellites of a uniform sky above 12 degrees, seen from p."""
    az = rng.uniform(0.0, 2.0 * np.pi, n)
    el = np.arcsin(rng.uniform(np.sin(np.radians(12.0)), np.sin(np.radians(88.0)), n))
    u = np.stack([np.cos(el) * np.sin(az), np.cos(el) * np.cos(az), np.sin(el)], 1) @ rot
    b = u @ p
    return p + (-b + np.sqrt(b * b - p @ p + ORBIT ** 2))[:, None] * u


def _circle(rng, speed):
    """(RING, 3) offsets and displacements (E/N/U, m) of a closed drive that
    starts and ends at the origin, 1 s per epoch."""
    th = rng.uniform(0.0, 2.0 * np.pi) + 2.0 * np.pi * np.arange(RING + 1) / RING
    r = speed * RING / (2.0 * np.pi)
    xy = r * np.stack([np.cos(th), np.sin(th)], 1)
    xy = np.concatenate([xy - xy[0], np.zeros((RING + 1, 1))], 1)
    return xy[1:], np.diff(xy, axis=0)


def _counts(case):
    """Particles per filter: log-uniform between n and n_max, fixed by the case."""
    f = case["filters"]
    if case["n_max"] == case["n"]:
        return np.full(f, case["n"], np.int64)
    r = np.random.default_rng(1000 + f)
    return np.exp(r.uniform(math.log(case["n"]), math.log(case["n_max"]), f)).astype(np.int64)


def _sat_counts(case):
    """(filters, RING) satellites in use, fixed by the case."""
    r = np.random.default_rng(2000 + case["filters"])
    return r.integers(case["sats_min"], case["sats"] + 1, (case["filters"], RING))


def _steps(case, seed):
    """Truth, clocks and per-epoch observations of every filter of a "step" case."""
    rng = np.random.default_rng(seed)
    base, rot = _frame()
    counts = _sat_counts(case)
    out = []
    for f in range(case["filters"]):
        start = base + (rng.uniform(-3000.0, 3000.0, 3) * [1, 1, 0]) @ rot
        off, disp = _circle(rng, rng.uniform(2.0, 20.0))
        clk = 3000.0 + rng.uniform(-50.0, 50.0, case["clocks"])
        sats = _sky(rng, start, rot, case["sats"])
        group = np.arange(case["sats"]) * case["clocks"] // case["sats"]
        epochs = []
        for t in range(RING):
            use = np.sort(rng.permutation(case["sats"])[: counts[f, t]])
            m = len(use)
            nlos = rng.random(m) < 0.2
            pr = np.linalg.norm(sats[use] - (start + off[t] @ rot), axis=1) + clk[group[use]]
            pr = pr + rng.normal(0.0, 3.0, m) + nlos * rng.exponential(15.0, m)
            cn0 = np.where(nlos, rng.normal(35.0, 5.0, m), rng.normal(45.0, 4.0, m))
            epochs.append(dict(disp=disp[t], sats=sats[use], pr=pr, w=rng.uniform(0.5, 1.0, m),
                               clk=group[use].astype(np.int32), cn0=cn0.astype(np.float32),
                               blocked=nlos.astype(np.float32)))
        out.append(SimpleNamespace(start=start, rot=rot, clk=clk, epochs=epochs, seed=int(rng.integers(1 << 31))))
    return out


NOISE = (1.0, 1.0, 0.5)      # predict noise of the "step" cases, E/N/U m
CLK_NOISE = 0.5
SPREAD, CLK_SPREAD = 3.0, 5.0


def _network(seed):
    """Parameters of the NLOS network (12-64-64-2, inputs padded to 16)."""
    r = np.random.default_rng(seed)
    w1 = r.normal(0.0, math.sqrt(2.0 / 12.0), (64, 16)) * (np.arange(16) < 12)
    w2 = r.normal(0.0, math.sqrt(2.0 / 64.0), (64, 64))
    w3 = r.normal(0.0, math.sqrt(1.0 / 64.0), (2, 64))
    return np.concatenate([w1.ravel(), np.zeros(64), w2.ravel(), np.zeros(64), w3.ravel(), [-1.0, 0.0]]).astype(np.float32)


def _device_inputs(case, seed):
    """Drive, satellites and pseudoranges of the single-filter kinds."""
    rng = np.random.default_rng(seed)
    start, rot = _frame()
    m = case.get("sats") or case["pairs"] + 2
    sats = _sky(rng, start, rot, m)
    off, disp = _circle(rng, 8.0)
    pos = start + off @ rot
    pr = np.linalg.norm(sats[None] - pos[:, None], axis=2) + 120.0 + rng.normal(0.0, 2.0, (RING, m))
    pr[:, : max(1, m // 5)] += rng.exponential(20.0, (RING, max(1, m // 5)))
    return SimpleNamespace(rng=rng, start=start, rot=rot, sats=sats, pos=pos, disp=disp, vel=disp @ rot, pr=pr,
                           w=rng.uniform(0.5, 1.0, m), seed=int(rng.integers(1 << 31)))


def _dd_results(case, d):
    """Double differences of every epoch: two constellations with a
    reference satellite each, a base station 4 km away."""
    base = d.start + np.array([2500.0, -3100.0, 5.0]) @ d.rot
    k = np.arange(2, case["pairs"] + 2)
    ref = k % 2
    br = np.linalg.norm(d.sats - base, axis=1)
    wl = np.where(ref == 0, WL, 0.24421021342456825)
    out = []
    for t in range(RING):
        r = np.linalg.norm(d.sats - d.pos[t], axis=1)
        dd = (r[k] - r[ref]) - (br[k] - br[ref])
        pr = dd + d.rng.normal(0.0, 0.6, len(k)) + (d.rng.random(len(k)) < 0.1) * d.rng.exponential(20.0, len(k))
        cy = dd / wl + d.rng.normal(0.0, 0.03, len(k)) + d.rng.integers(-40, 40, len(k))
        out.append(SimpleNamespace(n_dd=len(k), sat_ecef_k=d.sats[k], sat_ecef_ref=d.sats[ref],
                                   base_range_k=br[k], base_range_ref=br[ref], dd_weights=d.w[k],
                                   dd_pseudorange_m=pr, dd_carrier_cycles=cy, wavelengths_m=wl))
    return out


def _doppler_rows(d):
    """Satellite velocities and Doppler shifts of every epoch, receiver
    drift 30 m/s."""
    m = len(d.sats)
    u = d.rng.normal(size=(m, 3))
    sv = np.cross(u, d.sats)
    sv *= 3000.0 / np.linalg.norm(sv, axis=1, keepdims=True)
    out = []
    for t in range(RING):
        los = d.sats - d.pos[t]
        los /= np.linalg.norm(los, axis=1, keepdims=True)
        rate = np.sum((sv - d.vel[t]) * los, axis=1) + 30.0 + d.rng.normal(0.0, 0.15, m)
        out.append(-rate / WL)
    return sv, out


VEL = dict(sigma_pos=0.5, sigma_vel=0.4, init=1.0, q=0.2, sigma_mps=0.5, gain=0.25, cap=10.0)


def _records(case, seed):
    """Broadcast records, record index and times of an "orbits" case: Kepler
    records every 2 h, GLONASS states every 30 min."""
    rng = np.random.default_rng(seed)
    kep, glo, ne = case["kepler"], case["glonass"], case["epochs"]
    t = np.arange(ne, dtype=np.float64) * (86_400.0 / ne if ne < 2_880 else 1.0) + 18.0
    ks, gs = 12, 48
    system = np.array([ord("GGGGEEEJCC"[s % 10]) for s in range(kep)])
    k = {f: np.zeros((kep, ks)) for f in
         ("sqrt_a", "e", "i0", "omega0", "omega", "M0", "delta_n", "omega_dot", "idot", "cuc", "cus", "crc", "crs",
          "cic", "cis", "toe", "toc", "af0", "af1", "af2", "tgd")}
    k["sqrt_a"][:] = np.where(system == ord("C"), 5282.6, np.where(system == ord("E"), 5440.6, 5153.6))[:, None]
    for f, lo, hi in (("e", 1e-4, 0.02), ("i0", 0.9, 1.0), ("omega0", -3, 3), ("omega", -3, 3), ("M0", -3, 3),
                      ("af0", -1e-4, 1e-4), ("crc", 150, 300), ("crs", -60, 60), ("cuc", -4e-6, 4e-6),
                      ("cus", 2e-6, 9e-6), ("cic", -2e-7, 2e-7), ("cis", -2e-7, 2e-7), ("idot", -5e-10, 5e-10)):
        k[f][:] = rng.uniform(lo, hi, (kep, ks))
    k["delta_n"][:], k["omega_dot"][:], k["af1"][:], k["tgd"][:] = 4.5e-9, -8e-9, -1e-12, -1e-8
    k["toe"][:] = k["toc"][:] = 7200.0 * np.arange(ks) + 3600.0
    g = dict(toe=np.tile(1800.0 * np.arange(gs) + 900.0, (glo, 1)), pos=np.zeros((glo, gs, 3)),
             vel=np.zeros((glo, gs, 3)), acc=rng.uniform(-3e-6, 3e-6, (glo, gs, 3)),
             tau=rng.uniform(-2e-5, 2e-5, (glo, gs)), gam=rng.uniform(-1e-12, 1e-12, (glo, gs)))
    if glo:
        a = rng.uniform(0.0, 2.0 * np.pi, (glo, gs))
        v = math.sqrt(3.9860044e14 / 2.55e7)
        g["pos"][:] = 2.55e7 * np.stack([np.cos(a), np.sin(a), 0.0 * a], 2)
        g["vel"][:] = v * np.stack([-0.43 * np.sin(a), 0.43 * np.cos(a), 0.9 + 0.0 * a], 2)
    kj = np.clip(np.floor((t - 3600.0) / 7200.0 + 0.5), 0, ks - 1).astype(np.int32)
    gj = np.clip(np.floor((t - 918.0) / 1800.0 + 0.5), 0, gs - 1).astype(np.int32)
    idx = np.concatenate([np.arange(kep)[None] * ks + kj[:, None],
                          kep * ks + np.arange(glo)[None] * gs + gj[:, None]], 1).astype(np.int32)
    return SimpleNamespace(system=system, k=k, g=g, t=t, idx=idx, ks=ks, gs=gs)


def _train_set(case, seed):
    r = np.random.default_rng(seed)
    m = case["rows"]
    nlos = r.random(m) < 0.3
    el, az = r.uniform(0.2, 1.5, m), r.uniform(0.0, 2.0 * np.pi, m)
    rc = r.normal(0.0, 3.0, m) + nlos * r.exponential(20.0, m)
    x = np.stack([np.sin(el), np.cos(el), np.sin(az), np.cos(az), r.normal(0.3, 0.6, m) - nlos,
                  np.clip(rc / 20.0, -8, 8), np.minimum(np.abs(rc) / 20.0, 8), np.where(r.random(m) < 0.95, nlos, ~nlos),
                  r.integers(6, 41, m) / 40.0, r.uniform(0.05, 0.6, m), r.uniform(0.0, 0.6, m),
                  r.normal(0.0, 0.6, m) - nlos], 1)
    return x.astype(np.float32), np.stack([nlos, nlos * r.exponential(20.0, m)], 1).astype(np.float32)


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def _prepare_step(case, seed):
    from gnss_gpu_b200 import _native as N
    from gnss_gpu_b200.engine import Engine, EngineOptions, FilterSpec
    fl = _steps(case, seed)
    eng = Engine([FilterSpec(n_particles=int(n), seed=f.seed, sigma_pos=NOISE, sigma_clk=CLK_NOISE, sigma_pr=SIGMA_PR)
                  for n, f in zip(_counts(case), fl)],
                 EngineOptions(n_clk=case["clocks"], resampler=case["resampler"], megopolis_iters=case["iters"],
                               weight_mode=case["weight"], max_sats=case["sats"]))
    if case["weight"] == "mixture":
        eng.set_mlp(_network(seed))
    for k, f in enumerate(fl):
        eng.initialize(k, f.start, f.clk, SPREAD, CLK_SPREAD)
    flags = N.PF_EP_PREDICT | N.PF_EP_WEIGHT
    ring = [eng.pack_epoch([dict(f.epochs[t], flags=flags) for f in fl]) for t in range(RING)]
    return SimpleNamespace(kind="step", eng=eng, ring=ring, t=0)


def _prepare_device(case, seed):
    from gnss_gpu_b200 import ParticleFilterDevice
    d = _device_inputs(case, seed)
    pf = ParticleFilterDevice(n_particles=case["n"], sigma_pos=1.0, sigma_pr=SIGMA_PR, seed=d.seed,
                              nu=4.0 if case["likelihood"] == "student_t" else 0.0,
                              per_particle_huber=case["likelihood"] == "huber", per_particle_nlos_gate=case["gate"],
                              resampling=case["resampling"])
    pf.initialize(d.start, clock_bias=120.0, spread_pos=5.0, spread_cb=50.0)
    return SimpleNamespace(kind="device", pf=pf, d=d, gmm=case["likelihood"] == "gmm", t=0)


def _prepare_dd(case, seed):
    from gnss_gpu_b200 import ParticleFilterDevice
    d = _device_inputs(case, seed)
    pf = ParticleFilterDevice(n_particles=case["n"], sigma_pos=0.5, sigma_cb=1.0, seed=d.seed, resampling="systematic",
                              per_particle_nlos_gate=case["gate"], per_particle_huber=case["huber"])
    pf.initialize(d.start, clock_bias=120.0, spread_pos=2.0, spread_cb=5.0)
    return SimpleNamespace(kind="dd", pf=pf, d=d, dd=_dd_results(case, d), t=0)


def _prepare_doppler(case, seed):
    from gnss_gpu_b200 import _native as N
    from gnss_gpu_b200.engine import Engine, EngineOptions, FilterSpec
    d = _device_inputs(case, seed)
    sv, dop = _doppler_rows(d)
    eng = Engine([FilterSpec(n_particles=case["n"], seed=d.seed, sigma_pos=(0.0, 0.0, 0.0), sigma_clk=1.0,
                             sigma_pr=SIGMA_PR)],
                 EngineOptions(n_clk=1, weight_mode="generic", max_sats=case["sats"]))
    eng.initialize(0, d.start, 120.0, SPREAD, CLK_SPREAD)
    vel = eng.velocity_states(0)
    vel.init(d.vel[0], spread_vel=0.0, init_sigma=VEL["init"])
    weigh = [eng.pack_epoch([dict(disp=np.zeros(3), sats=d.sats, pr=d.pr[t], w=d.w,
                                  flags=N.PF_EP_PREDICT | N.PF_EP_WEIGHT | N.PF_EP_NO_RESAMPLE)]) for t in range(RING)]
    check = eng.pack_epoch([dict(disp=np.zeros(3), flags=N.PF_EP_RESAMPLE_CHECK)])
    return SimpleNamespace(kind="doppler", eng=eng, vel=vel, d=d, sv=sv, dop=dop, weigh=weigh, check=check,
                           kf=case["kf"], t=0)


def _prepare_city(case, seed):
    from gnss_gpu_b200 import BVHAccelerator, ParticleFilter3DBVH
    from gnss_gpu_b200 import citysim as CS
    rng = np.random.default_rng(seed)
    base, rot = _frame()
    city = CS.make_city(int(rng.integers(1 << 30)), size=2000.0, cell=case["cell"])
    bvh = BVHAccelerator(CS.city_triangles(city, base, rot))
    # a drive around a street crossing near the centre (block edges are streets)
    cross = np.round(rng.uniform(600.0, 1400.0, 2) / case["cell"]) * case["cell"]
    start = base + np.array([cross[0], cross[1], 1.5]) @ rot
    off, disp = _circle(rng, 2.0)
    sats = _sky(rng, start, rot, case["sats"])
    pos = start + off @ rot
    pr = np.linalg.norm(sats[None] - pos[:, None], axis=2) + 80.0 + rng.normal(0.0, 1.0, (RING, case["sats"]))
    for t in range(RING):
        pr[t] += np.where(bvh.check_los(pos[t], sats), 0.0, 25.0)
    pf = ParticleFilter3DBVH(bvh, n_particles=case["n"], sigma_pos=0.5, sigma_cb=1.0, sigma_pr=3.0,
                             resampling="systematic", seed=int(rng.integers(1 << 31)))
    pf.initialize(start, 80.0, case["spread"], 5.0)
    return SimpleNamespace(kind="city", pf=pf, sats=sats, pr=pr, vel=disp @ rot, w=np.ones(case["sats"]), t=0)


def _prepare_orbits(case, seed):
    from gnss_gpu_b200 import _native as N
    o = _records(case, seed)
    kep, glo = case["kepler"], case["glonass"]
    rec = np.zeros(kep * o.ks + glo * o.gs, N.BROADCAST_DTYPE)
    rec["system"] = np.concatenate([np.repeat(o.system, o.ks), np.full(glo * o.gs, ord("R"))])
    for f, v in o.k.items():
        rec["kepler"][f][: kep * o.ks] = v.ravel()
    if glo:
        g = rec["glonass"]
        for f, v in (("toe", "toe"), ("pos", "pos"), ("vel", "vel"), ("acc", "acc"), ("tau_n", "tau"),
                     ("gamma_n", "gam")):
            g[f][kep * o.ks:] = o.g[v].reshape((glo * o.gs,) + o.g[v].shape[2:])
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    ne, ns = o.idx.shape
    return SimpleNamespace(kind="orbits", lib=N.load(), check=N.check, n_rec=len(rec), rec=up(rec.view(np.uint8)),
                           idx=up(o.idx), t=up(o.t), ne=ne, ns=ns,
                           pos=torch.empty((ne, ns, 3), dtype=torch.float64, device="cuda"),
                           clk=torch.empty((ne, ns), dtype=torch.float64, device="cuda"))


def _prepare_train(case, seed):
    from gnss_gpu_b200 import _native as N
    lib = N.load()
    x, y = _train_set(case, seed)
    prm = torch.from_numpy(_network(seed)).cuda()
    return SimpleNamespace(kind="train", lib=lib, check=N.check, rows=case["rows"], x=torch.from_numpy(x).cuda(),
                           y=torch.from_numpy(y).cuda(), prm=prm, m=torch.zeros_like(prm), v=torch.zeros_like(prm),
                           loss=torch.zeros(1, device="cuda"), step=0,
                           scratch=torch.zeros(lib.pf_mlp_scratch_bytes(), dtype=torch.uint8, device="cuda"))


_PREPARE = dict(step=_prepare_step, device=_prepare_device, dd=_prepare_dd, doppler=_prepare_doppler,
                city=_prepare_city, orbits=_prepare_orbits, train=_prepare_train)


# --------------------------------------------------------------------- run
def run(s):
    return _RUN[s.kind](s)


def _results(r):
    f4 = np.float32
    return dict(est=r["est_ecef"].copy(), clk=r["est_clk"].astype(f4), cov=r["cov_enu"].astype(f4),
                ess=r["ess"].astype(f4), sum_w=r["sum_w"].astype(f4), resampled=r["resampled"].copy())


def _run_step(s):
    fe, sats = s.ring[s.t % RING]
    s.t += 1
    return _results(np.ctypeslib.as_array(s.eng.step_io(fe, sats)))


def _run_device(s):
    t = s.t % RING
    s.t += 1
    s.pf.predict(s.d.vel[t], dt=1.0)
    if s.gmm:
        s.pf.update_gmm(s.d.sats, s.d.pr[t], s.d.w)
    else:
        s.pf.update(s.d.sats, s.d.pr[t], s.d.w)
    e = s.pf.estimate()
    return dict(est=e[:3], clk=e[3:].astype(np.float32))


def _run_dd(s):
    t = s.t % RING
    s.t += 1
    s.pf.predict(s.d.vel[t], dt=1.0)
    s.pf.update_dd_pseudorange(s.dd[t], sigma_pr=0.75, resample=False)
    s.pf.update_dd_carrier_afv(s.dd[t], sigma_cycles=0.1, resample=False)
    e, ess = s.pf.estimate(), s.pf.get_ess()
    return dict(est=e[:3], ess=np.float32(ess), resampled=int(s.pf.resample_if_needed()))


def _run_doppler(s):
    t = s.t % RING
    s.t += 1
    s.vel.predict(s.d.vel[t], 1.0, VEL["sigma_pos"], VEL["sigma_vel"], 0.5, s.kf, VEL["q"], s.t)
    s.eng.upload(0, *s.weigh[t])
    s.eng.step()
    s.vel.doppler(s.d.sats, s.sv, s.dop[t], s.d.w, WL, VEL["sigma_mps"], VEL["gain"], VEL["cap"], kf=s.kf)
    s.eng.upload(0, *s.check)
    s.eng.step()
    r = _results(s.eng.results_array())
    # the velocity states as the Doppler update left them: the resample is
    # applied to them when they are next used
    k = s.vel.NCOMP * s.vel.n
    now = s.vel.buf[s.vel.vs.sel * k:(s.vel.vs.sel + 1) * k].view(s.vel.NCOMP, s.vel.n)
    return dict(r, vel=now[:3], var=now[3:])


def _run_city(s):
    t = s.t % RING
    s.t += 1
    s.pf.predict(s.vel[t], dt=1.0)
    s.pf.update(s.sats, s.pr[t], s.w)
    r = s.pf.last_step()
    return dict(est=r["est_ecef"], clk=r["est_clk"].astype(np.float32), cov=r["cov_enu"].astype(np.float32),
                ess=np.float32(r["ess"]), resampled=int(r["resampled"]))


def _run_orbits(s):
    st = torch.cuda.current_stream().cuda_stream
    s.check(s.lib.pf_broadcast_orbits(s.rec.data_ptr(), s.n_rec, s.idx.data_ptr(), s.t.data_ptr(), s.ne, s.ns, 60.0,
                                      s.pos.data_ptr(), s.clk.data_ptr(), st))
    return dict(pos=s.pos, clk=s.clk)


def _run_train(s):
    s.step += 1
    st = torch.cuda.current_stream().cuda_stream
    s.check(s.lib.pf_mlp_adam_step(s.x.data_ptr(), s.y.data_ptr(), s.rows, s.prm.data_ptr(), s.m.data_ptr(),
                                   s.v.data_ptr(), s.step, 2e-3, s.loss.data_ptr(), s.scratch.data_ptr(),
                                   s.scratch.numel(), st))
    return dict(prm=s.prm, m=s.m, v=s.v, loss=s.loss)


_RUN = dict(step=_run_step, device=_run_device, dd=_run_dd, doppler=_run_doppler, city=_run_city, orbits=_run_orbits,
            train=_run_train)


# -------------------------------------------------------------------- work
def work(case):
    """Bytes: the particle state (FP32 components, log-weight, ancestor;
    FP64 velocity states) read once and written once, inputs and results.
    Operations: draws and motion, the likelihood terms, the statistics (a
    square root, divide, logarithm or sine counted as one)."""
    kind = case["kind"]
    if kind == "step":
        n, s = _counts(case).astype(float), _sat_counts(case).mean(1)
        d = 3 + case["clocks"]
        term = {"gaussian": 18, "huber": 22, "mixture": 30}[case["weight"]]
        flops = n * (60.0 * d + term * s + 40.0)
        if case["resampler"] == "megopolis":
            flops = flops + n * 8.0 * case["iters"]
        return dict(bytes=float(np.sum(n * (8.0 * d + 12.0) + 56.0 * s)), flops=float(np.sum(flops)))
    if kind == "train":
        m = case["rows"]
        return dict(bytes=56.0 * m + 24.0 * 5378, flops=3.0 * 2.0 * m * (12 * 64 + 64 * 64 + 64 * 2))
    if kind == "orbits":
        m = float(case["epochs"])
        return dict(bytes=m * (case["kepler"] + case["glonass"]) * 36.0 + 8.0 * m,
                    flops=m * (case["kepler"] * 130.0 + case["glonass"] * 330.0))
    n = float(case["n"])
    if kind == "device":
        return dict(bytes=n * 44.0, flops=n * (240.0 + case["sats"] * 22.0 * (2 if case["gate"] else 1) + 40.0))
    if kind == "dd":
        return dict(bytes=n * 44.0, flops=n * (240.0 + 2 * case["pairs"] * 24.0 + 40.0))
    if kind == "doppler":
        per = 160.0 if case["kf"] else 90.0
        return dict(bytes=n * (44.0 + 16.0 * (12 if case["kf"] else 3)), flops=n * (400.0 + case["sats"] * (per + 20.0)))
    return dict(bytes=n * 44.0, flops=n * (240.0 + case["sats"] * 60.0))  # city: ranges, likelihood, the rays' set-up


# ------------------------------------------------------------------- exact
def exact(case, seed):
    kind = case["kind"]
    if kind == "step" and case["weight"] != "mixture":
        return _exact_step(case, seed)
    if kind == "dd":
        return _exact_dd(case, seed)
    if kind == "doppler":
        return _exact_doppler(case, seed)
    if kind == "orbits":
        return _exact_orbits(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    # mixture: a BF16 network decides each satellite's likelihood; device:
    # the estimate follows the random resample; city: the particles' order
    # (and with it each one's noise) follows from their FP32 positions
    return None


def _dev(a):
    return torch.as_tensor(np.asarray(a, np.float64), device="cuda")


def _philox(n, c1, tag, fid, seed):
    """Philox4x32-10 (Salmon et al., SC'11) at counters (0..n-1, c1, tag, fid)."""
    m32 = 0xFFFFFFFF
    c = [torch.arange(n, dtype=torch.int64, device="cuda")] + [torch.full((n,), v, dtype=torch.int64, device="cuda")
                                                               for v in (c1, tag, fid)]
    k0, k1 = seed & m32, seed >> 32
    for _ in range(10):
        p, q = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
        c = [((q >> 32) & m32) ^ c[1] ^ k0, q & m32, ((p >> 32) & m32) ^ c[3] ^ k1, p & m32]
        k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
    return [v.double() for v in c]


def _normals(n, c1, tag, fid, seed, count, top24=True):
    """`count` standard normals per particle, four per Philox block
    (Box-Muller; top24: the angle from the upper 24 bits of its word)."""
    z = []
    for b in range((count + 3) // 4):
        r = _philox(n, c1, tag | b, fid, seed)
        for u, v in ((r[0], r[1]), (r[2], r[3])):
            rad = torch.sqrt(-2.0 * torch.log((u + 0.5) * 2.0 ** -32))
            ang = 2.0 * math.pi * ((torch.floor(v / 256.0) * 2.0 ** -24 if top24 else v * 2.0 ** -32) - 0.5)
            z += [rad * torch.cos(ang), rad * torch.sin(ang)]
    return torch.stack(z[:count], 1)


TAG_INIT, TAG_PREDICT, TAG_VEL_PREDICT = 0x01000000, 0x02000000, 0x07000000


def _cloud(n, fid, seed, clocks, spread, spread_clk):
    z = _normals(n, 0, TAG_INIT, fid, seed, 3 + clocks)
    return spread * z[:, :3], spread_clk * z[:, 3:]


def _stats(x, clk, lw, start, rot, clk0, n):
    """Weighted mean, covariance, ESS and sum of the weights."""
    w = torch.exp(lw - lw.max())
    sw = w.sum()
    mu, mc = (w[:, None] * x).sum(0) / sw, (w[:, None] * clk).sum(0) / sw
    xc = x - mu
    cov = torch.stack([(w * xc[:, i] * xc[:, j]).sum() / sw for i, j in
                       ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))])
    ess = float(sw * sw / (w * w).sum())
    c = np.zeros(4)
    c[: len(clk0)] = np.asarray(clk0) + mc.cpu().numpy()
    return dict(est=start + mu.cpu().numpy() @ rot, clk=c, cov=cov.cpu().numpy(), ess=ess, sum_w=float(sw))


def _pseudorange_lw(x, clk, sats, pr, w, group, start, rot, clk0, huber=None):
    p = _dev(start) + x @ _dev(rot)
    lw = torch.zeros(len(x), dtype=torch.float64, device="cuda")
    for j in range(len(pr)):
        r = pr[j] - torch.linalg.norm(_dev(sats[j]) - p, dim=1) - (clk0[group[j]] + clk[:, group[j]])
        z = r.abs() / SIGMA_PR
        rho = 0.5 * z * z
        if huber:
            rho = torch.where(z < huber, rho, huber * z - 0.5 * huber * huber)
        lw -= w[j] * rho
    return lw


def _exact_step(case, seed):
    out = {k: [] for k in ("est", "clk", "cov", "ess", "sum_w")}
    for k, (n, f) in enumerate(zip(_counts(case), _steps(case, seed))):
        n, e = int(n), f.epochs[0]
        x, c = _cloud(n, k, f.seed, case["clocks"], SPREAD, CLK_SPREAD)
        z = _normals(n, 0, TAG_PREDICT, k, f.seed, 3 + case["clocks"])
        x = x + _dev(e["disp"]) + _dev(NOISE) * z[:, :3]
        c = c + CLK_NOISE * z[:, 3:]
        lw = _pseudorange_lw(x, c, e["sats"], e["pr"], e["w"], e["clk"], f.start, f.rot, f.clk,
                             1.5 if case["weight"] == "huber" else None)
        s = _stats(x, c, lw, f.start, f.rot, f.clk, n)
        for q in out:
            out[q].append(s[q])
    return dict({q: np.array(v) for q, v in out.items()}, resampled=None)


def _dd_lw(x, r, sigma, wl, gate, huber, start, rot, obs):
    """Log-likelihood of double differences (fractional cycles when wl is given)."""
    p = _dev(start) + x @ _dev(rot)
    dist = lambda s: torch.linalg.norm(_dev(s) - p, dim=1)  # noqa: E731
    v = []
    for j in range(r.n_dd):
        d = dist(r.sat_ecef_k[j]) - dist(r.sat_ecef_ref[j]) - r.base_range_k[j] + r.base_range_ref[j]
        d = obs[j] - (d if wl is None else d / wl[j])
        v.append(d if wl is None else d - torch.round(d))
    v = torch.stack(v, 1)
    z = v.abs() / sigma
    rho = 0.5 * z * z
    if huber:
        rho = torch.where(z < huber, rho, huber * z - 0.5 * huber * huber)
    rho = rho * _dev(r.dd_weights)
    if gate:
        inside = v.abs() <= gate
        rho = torch.where((inside.sum(1, keepdim=True) >= min(3, r.n_dd)) & ~inside, torch.zeros_like(rho), rho)
    return -rho.sum(1)


def _exact_dd(case, seed):
    d = _device_inputs(case, seed)
    r = _dd_results(case, d)[0]
    n = case["n"]
    x, c = _cloud(n, 0, d.seed, 1, 2.0, 5.0)
    z = _normals(n, 0, TAG_PREDICT, 0, d.seed, 4)
    x = x + _dev(d.rot @ d.vel[0]) + 0.5 * z[:, :3]
    hk = 1.5 if case["huber"] else None
    lw = _dd_lw(x, r, 0.75, None, 10.0 if case["gate"] else None, hk, d.start, d.rot, r.dd_pseudorange_m)
    lw = lw + _dd_lw(x, r, 0.1, r.wavelengths_m, 0.5 if case["gate"] else None, hk, d.start, d.rot, r.dd_carrier_cycles)
    s = _stats(x, c, lw, d.start, d.rot, [120.0], n)
    return dict(est=s["est"], ess=s["ess"], resampled=None)


def _exact_doppler(case, seed):
    d = _device_inputs(case, seed)
    sv, dop = _doppler_rows(d)
    n, kf = case["n"], case["kf"]
    x, c = _cloud(n, 0, d.seed, 1, SPREAD, CLK_SPREAD)
    z = _normals(n, 1, TAG_VEL_PREDICT, 0, d.seed, 8, top24=False)
    v = _dev(d.vel[0]).expand(n, 3).clone()
    P = VEL["init"] ** 2 * torch.eye(3, dtype=torch.float64, device="cuda").expand(n, 3, 3).clone()
    v = 0.5 * v + 0.5 * _dev(d.vel[0])
    if kf:
        nz = z[:, :3] * math.sqrt(VEL["sigma_pos"] ** 2 + VEL["init"] ** 2)
        P = P + VEL["q"] * torch.eye(3, dtype=torch.float64, device="cuda")
    else:
        v = v + VEL["sigma_vel"] * z[:, :3]
        nz = VEL["sigma_pos"] * z[:, 3:6]
    x = x + (v + nz) @ _dev(d.rot).T
    c = c + 1.0 * _normals(n, 0, TAG_PREDICT, 0, d.seed, 4)[:, 3:4]
    lw = _pseudorange_lw(x, c, d.sats, d.pr[0], d.w, np.zeros(len(d.w), int), d.start, d.rot, [120.0])
    p = _dev(d.start) + x @ _dev(d.rot)
    los = _dev(d.sats)[None] - p[:, None]
    los = los / torch.linalg.norm(los, dim=2, keepdim=True)
    w = _dev(d.w)
    y = -_dev(dop[0]) * WL - (los * _dev(sv)).sum(2)     # rate with the satellite's part taken out
    if kf:
        hm = (w[None, :, None] * -los).sum(1) / w.sum()
        ym = (w * y).sum(1) / w.sum()
        for j in range(len(dop[0])):
            h = -los[:, j] - hm
            ph = torch.einsum("nij,nj->ni", P, h)
            S = (h * ph).sum(1) + VEL["sigma_mps"] ** 2 / w[j]
            innov = y[:, j] - ym - (h * v).sum(1)
            K = ph / S[:, None]
            v = v + K * innov[:, None]
            P = P - K[:, :, None] * ph[:, None, :]
            P = 0.5 * (P + P.transpose(1, 2))
            lw = lw - 0.5 * (innov * innov / S + torch.log(S))
    else:
        cd = (w * (y + (los * v[:, None]).sum(2))).sum(1) / w.sum()
        res = y + (los * v[:, None]).sum(2) - cd[:, None]
        lw = lw - 0.5 * (w * res * res).sum(1) / VEL["sigma_mps"] ** 2
        H = torch.cat([-los, torch.ones_like(los[:, :, :1])], 2)
        A = torch.einsum("nsi,s,nsj->nij", H, w, H) + 1e-9 * torch.eye(4, dtype=torch.float64, device="cuda")
        sol = torch.linalg.solve(A, torch.einsum("nsi,s,ns->ni", H, w, y))
        dv = sol[:, :3] - v
        nrm = torch.linalg.norm(dv, dim=1, keepdim=True)
        v = v + VEL["gain"] * torch.where(nrm > VEL["cap"], dv * VEL["cap"] / nrm, dv)
    s = _stats(x, c, lw, d.start, d.rot, [120.0], n)
    return dict({k: np.array([q]) for k, q in s.items()}, resampled=None, vel=v.T.contiguous(),
                var=P.reshape(n, 9).T.contiguous())


def _exact_orbits(case, seed):
    o = _records(case, seed)
    t = _dev(o.t)[:, None]
    col = lambda a, j: _dev(a.reshape(-1))[torch.as_tensor(j, device="cuda").long()]  # noqa: E731
    kep = case["kepler"]
    k = {f: col(v, o.idx[:, :kep]) for f, v in o.k.items()}
    sysm = o.system
    mu = _dev(np.where((sysm == ord("E")) | (sysm == ord("C")), 3.986004418e14, 3.986005e14))
    we = _dev(np.where(sysm == ord("C"), 7.292115e-5, 7.2921151467e-5))
    rel = _dev(np.where((sysm == ord("E")) | (sysm == ord("C")), -4.442807309e-10, -4.442807633e-10))
    rx = t - _dev(np.where(sysm == ord("C"), 14.0, 0.0))
    rx = torch.where(rx < 0, rx + 604800.0, rx)
    half = lambda d: torch.where(d > 302400.0, d - 604800.0, torch.where(d < -302400.0, d + 604800.0, d))  # noqa: E731
    a = k["sqrt_a"] ** 2
    tk = half(rx - k["toe"])
    M = k["M0"] + (torch.sqrt(mu / a ** 3) + k["delta_n"]) * tk
    E = M.clone()
    for _ in range(12):
        E = E + (M - E + k["e"] * torch.sin(E)) / (1.0 - k["e"] * torch.cos(E))
    sE, cE = torch.sin(E), torch.cos(E)
    phi = torch.atan2(torch.sqrt(1.0 - k["e"] ** 2) * sE, cE - k["e"]) + k["omega"]
    s2, c2 = torch.sin(2 * phi), torch.cos(2 * phi)
    u = phi + k["cuc"] * c2 + k["cus"] * s2
    r = a * (1.0 - k["e"] * cE) + k["crc"] * c2 + k["crs"] * s2
    inc = k["i0"] + k["idot"] * tk + k["cic"] * c2 + k["cis"] * s2
    Om = k["omega0"] + (k["omega_dot"] - we) * tk - we * k["toe"]
    xp, yp = r * torch.cos(u), r * torch.sin(u)
    pos = torch.stack([xp * torch.cos(Om) - yp * torch.cos(inc) * torch.sin(Om),
                       xp * torch.sin(Om) + yp * torch.cos(inc) * torch.cos(Om), yp * torch.sin(inc)], 2)
    dt = half(rx - k["toc"])
    clk = k["af0"] + k["af1"] * dt + k["af2"] * dt * dt + rel * k["e"] * k["sqrt_a"] * sE - k["tgd"]
    if case["glonass"]:
        j = o.idx[:, kep:] - kep * o.ks
        g = {f: _dev(v.reshape((-1,) + v.shape[2:]))[torch.as_tensor(j, device="cuda").long()] for f, v in o.g.items()}
        rx = t - 18.0
        rx = torch.where(rx < 0, rx + 604800.0, rx)
        el = half(rx - g["toe"])
        x = torch.cat([g["pos"], g["vel"]], 2)
        we, gmu, j2, re = 7.292115e-5, 3.9860044e14, 1.0826257e-3, 6378136.0

        def f(x):
            r2 = (x[..., :3] ** 2).sum(-1)
            r3 = r2 * torch.sqrt(r2)
            at = 1.5 * j2 * gmu * re ** 2 / r2 / r3
            ct = -gmu / r3 - at * (1.0 - 5.0 * x[..., 2] ** 2 / r2)
            acc = torch.stack([(ct + we * we) * x[..., 0] + 2 * we * x[..., 4],
                               (ct + we * we) * x[..., 1] - 2 * we * x[..., 3], (ct - 2 * at) * x[..., 2]], -1)
            return torch.cat([x[..., 3:], acc + g["acc"]], -1)

        rem = el.clone()
        while bool((rem.abs() > 1e-9).any()):
            h = torch.where(rem.abs() >= 60.0, 60.0 * torch.sign(rem), torch.where(rem.abs() > 1e-9, rem, 0.0 * rem))
            hh = h[..., None]
            k1 = f(x)
            k2 = f(x + k1 * hh / 2)
            k3 = f(x + k2 * hh / 2)
            x = x + (k1 + 2 * k2 + 2 * k3 + f(x + k3 * hh)) * hh / 6
            rem = rem - h
        pos = torch.cat([pos, x[..., :3]], 1)
        clk = torch.cat([clk, -g["tau"] + g["gam"] * el], 1)
    return dict(pos=pos, clk=clk)


def _exact_train(case, seed):
    x, y = _train_set(case, seed)
    x, y = _dev(x), _dev(y)
    p = _dev(_network(seed)).requires_grad_(True)
    w1, b1 = p[:1024].view(64, 16)[:, :12], p[1024:1088]
    w2, b2 = p[1088:5184].view(64, 64), p[5184:5248]
    w3, b3 = p[5248:5376].view(2, 64), p[5376:]
    o = torch.relu(torch.relu(x @ w1.T + b1) @ w2.T + b2) @ w3.T + b3
    bce = torch.nn.functional.binary_cross_entropy_with_logits(o[:, 0], y[:, 0])
    loss = bce + (y[:, 0] * (torch.nn.functional.softplus(o[:, 1]) - y[:, 1] / 20.0) ** 2).mean()
    g, = torch.autograd.grad(loss, p)
    m, v = 0.1 * g, 0.001 * g * g
    prm = p.detach() - 2e-3 * (m / 0.1) / (torch.sqrt(v / 0.001) + 1e-8)
    return dict(prm=prm, m=m, v=v, loss=loss.detach()[None])
