"""Kernel launches that the driver refuses, made on the host: the library runs in a
child process against a CUDA runtime without a GPU (tests/fake_cudart.c), which
refuses the chosen call.  The library's call returns an error and leaves the
filter as it was."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent

CHILD = r"""
import ctypes as C, json, sys
fake = C.CDLL(sys.argv[1], mode=C.RTLD_GLOBAL)
fake.fake_log.restype = C.c_char_p
sys.path.insert(0, sys.argv[2])
import numpy as np
from gnss_gpu_b200 import _native as N
assert "torch" not in sys.modules   # it would bring the real runtime
L = N.load()
n, out = 40_003, {}


def launched(name):
    return fake.fake_log().decode().count(name)


def block(nbytes):   # 256-byte aligned memory
    raw = C.create_string_buffer(nbytes + 256)
    at = (C.addressof(raw) + 255) & ~255
    keep.append(raw)
    return C.c_void_p(at)


keep = []
cfg = N.EngineConfig(n_filters=1, n_clk=1, resampler=0, megopolis_iters=15, weight_mode=0, lw_mode=0, sys_offset=0,
                     max_sats=16, obs_slots=1, flags=3, ess_threshold=0.5, huber_k=1.5)
prm = (N.FilterParams * 1)()
prm[0].n_particles, prm[0].seed, prm[0].sigma_clk, prm[0].sigma_pr = n, 3, 1.0, 3.0
need, h, stream = C.c_size_t(0), C.c_void_p(), block(64)
N.check(L.pfe_workspace_bytes(C.byref(cfg), prm, C.byref(need)))
N.check(L.pfe_create(C.byref(cfg), prm, block(need.value), need, stream, C.byref(h)))
p0, clk = np.array([-3957199.0, 3310205.0, 3737911.0]), np.zeros(4)
N.check(L.pfe_initialize(h, 0, N.dptr(p0), N.dptr(clk), 5.0, 3.0))


def control(**change):
    # the five last words of the control block: rs_seq, resample_flag, lw_zero, parity, initialized
    size = C.c_size_t(0)
    N.check(L.pfe_checkpoint_bytes(h, 0, C.byref(size)))
    blob = np.zeros(size.value, np.uint8)
    N.check(L.pfe_checkpoint_save(h, 0, N.vptr(blob), size))
    nctrl = int(blob[24:28].view(np.int32)[0])
    words = blob[32 + 72:32 + 72 + nctrl].view(np.int32)
    at = [i for i in range(len(words) - 4) if words[i + 4] == 1 and not words[i + 5:].any()][-1]
    w = words[at:at + 5]
    for k, v in change.items():
        w[["rs_seq", "resample_flag", "lw_zero", "parity"].index(k)] = v
    if change:
        N.check(L.pfe_checkpoint_load(h, 0, N.vptr(blob), size))
    return [int(x) for x in w]


def refused(part, call):
    fake.fake_clear_log()
    fake.fake_refuse(part.encode())
    status = call()
    fake.fake_refuse(b"")
    return status


SCENARIO
print(json.dumps(out))
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    d = tmp_path_factory.mktemp("fake_cudart")
    so, ver = d / "libcudart.so.12", d / "version"
    ver.write_text("libcudart.so.12 { global: *; };\n")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-Wl,-soname,libcudart.so.12", f"-Wl,--version-script={ver}",
                    str(HERE / "fake_cudart.c"), "-o", str(so)], check=True)
    return so


def run(fake, scenario):
    src = CHILD.replace("SCENARIO", scenario)
    r = subprocess.run([sys.executable, "-c", src, str(fake), str(HERE.parent)], capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0, r.stderr
    return json.loads(r.stdout.splitlines()[-1])


PREDICT = r"""
vs = N.VelState()
vs.buf = block(2 * 12 * n * 8)
vs.sel, vs.seq = 0, 7
out["control"] = control(resample_flag=1, rs_seq=9)
g = np.zeros(3)
predict = lambda: L.pfe_vel_predict(h, 0, C.byref(vs), N.dptr(g), 1.0, 0.5, 0.1, 0.5, 0, 0.0, 1)
"""


def test_velocity_predict_refused(fake):
    """The filter keeps its buffer and its pending resample, the velocity state its
    buffer; the next call follows the resample as if nothing had been."""
    r = run(fake, PREDICT + r"""
out["status"] = refused("k_vel_predict", predict)
out["flips"], out["state"], out["after"] = launched("k_flip_state"), [vs.sel, vs.seq], control()
out["again"] = predict()
out["state_again"] = [vs.sel, vs.seq]
""")
    assert r["status"] != 0 and r["flips"] == 0
    assert r["state"] == [0, 7] and r["after"] == r["control"]
    assert r["again"] == 0 and r["state_again"] == [1, 9]


RAYS = r"""
mesh = N.Mesh()
mesh.nodes, mesh.tris, mesh.n_nodes, mesh.n_tris = block(64), block(64), 1, 1
def term(n_sat):
    sats = np.zeros(5 * n_sat)
    return L.pfe_add_3d_term(h, 0, C.byref(mesh), N.dptr(sats), n_sat, 3.0, 30.0, 10.0, 0.8, 0.1, 0)
out["base"], out["lw_zero"] = fake.fake_pool_blocks(), control()[2]
N.check(term(1)); out["words"] = launched("k_rays_3d")
N.check(term(64)); out["cells"] = launched("k_cells_cell")
out["ok"] = fake.fake_pool_blocks()
"""


@pytest.mark.parametrize("n_sat,part", [(1, "k_rays_3d"), (1, "k_weight_3d"), (64, "k_cells_box"), (64, "k_cells_mark"),
                                        (64, "k_cells_block"), (64, "k_cells_cell"), (64, "k_weight_3d"), (64, "fill")])
def test_ray_scratch_goes_back_when_a_kernel_is_refused(fake, n_sat, part):
    r = run(fake, RAYS + f"""
fake.fake_refuse_fill(int("{part}" == "fill"))
out["status"] = [refused("{part}" if "{part}" != "fill" else "", lambda: term({n_sat})) for _ in range(3)]
fake.fake_refuse_fill(0)
out["done"] = launched("k_term_done")
out["later"] = fake.fake_log().decode().splitlines()
out["after"] = fake.fake_pool_blocks()
out["again"] = term({n_sat})
""")
    assert r["words"] == 1 and r["cells"] == 1 and r["ok"] == r["base"]  # both routes were taken
    assert all(r["status"]) and r["done"] == 0 and r["again"] == 0
    assert r["after"] == r["base"]
    chain = ["k_rays_3d", "k_weight_3d"] if n_sat == 1 else ["k_cells_box", "k_cells_mark", "k_cells_block",
                                                              "k_cells_cell", "k_weight_3d", "k_weight_3d"]
    before = chain[:chain.index(part)] if part != "fill" else []
    assert len(r["later"]) == len(before) and all(b in ln for b, ln in zip(before, r["later"]))


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("rows", [4, 40])
def test_observation_term_refused(fake, kind, rows):
    """The log-weights stay read as zero, as before the call."""
    r = run(fake, f"""
rows = np.zeros({rows}, N.OBS_ROW_DTYPE)
rows["weight"], rows["wavelength"] = 1.0, 0.19
term = lambda: L.pfe_add_obs_term(h, 0, {kind}, N.vptr(rows), {rows}, 1.0, 0.0, 0.0, 0)
out["status"], out["done"], out["again"] = refused("k_obs_term", term), launched("k_term_done"), term()
out["done_again"] = launched("k_term_done")
""")
    assert r["status"] != 0 and r["done"] == 0
    assert r["again"] == 0 and r["done_again"] == 1


@pytest.mark.parametrize("part", ["k_glo_need", "k_glo_table", "k_broadcast_orbits", "fill"])
def test_orbits_refused(fake, part):
    """No later kernel runs on a table that was not made, and the scratch goes back."""
    r = run(fake, f"""
rec = np.zeros(4, N.BROADCAST_DTYPE)
rec["system"] = ord("R")
t, pos, clk = np.arange(100.0), np.zeros((100, 4, 3)), np.zeros((100, 4))
orbits = lambda: L.pf_broadcast_orbits(N.vptr(rec), 4, None, N.vptr(t), 100, 4, 60.0, N.vptr(pos), N.vptr(clk), None)
N.check(orbits())
out["chain"], out["base"] = fake.fake_log().decode().splitlines()[-3:], fake.fake_pool_blocks()
fake.fake_refuse_fill(int("{part}" == "fill"))
out["status"] = refused("{part}" if "{part}" != "fill" else "", orbits)
fake.fake_refuse_fill(0)
out["ran"], out["after"], out["again"] = fake.fake_log().decode().splitlines(), fake.fake_pool_blocks(), orbits()
""")
    names = ["k_glo_need", "k_glo_table", "k_broadcast_orbits"]
    assert len(r["chain"]) == 3 and all(n in ln for n, ln in zip(names, r["chain"]))
    before = names[:names.index(part)] if part != "fill" else []
    assert r["status"] != 0 and len(r["ran"]) == len(before)
    assert r["after"] == r["base"] and r["again"] == 0


def test_results_behind_a_step_and_on_an_idle_stream(fake):
    """The control blocks come by a kernel behind a step in flight, by the copy engine
    when nothing is: the same results."""
    r = run(fake, r"""
res, ess = (N.FilterResult * 1)(), C.c_double(0)
for step in (0, 1):
    for name, read in (("results", lambda: L.pfe_read_results(h, res)), ("ess", lambda: L.pfe_get_ess(h, 0, C.byref(ess)))):
        if step:
            N.check(L.pfe_step(h))
        fake.fake_clear_log()
        out[f"{name}{step}"] = [read(), launched("k_mirror"), res[0].initialized, ess.value]
""")
    assert r["results0"] == [0, 0, 1, 0.0] and r["results1"] == [0, 1, 1, 40_003.0]
    assert r["ess0"] == [0, 0, 1, 40_003.0] and r["ess1"] == [0, 1, 1, 40_003.0]


def test_only_the_one_call_step_carries_its_records(fake):
    """A step whose records are in the ring launches the kernel without the 3.7 KB
    parameter; the one-call step takes it where the records fit."""
    r = run(fake, r"""
fe, sats = np.zeros(1, N.FILTER_EPOCH_DTYPE), np.zeros(16, N.SAT_DTYPE)
res = (N.FilterResult * 1)()
for name, call in (("step", lambda: L.pfe_step(h)), ("per_filter", lambda: L.pfe_step_per_filter(h)),
                   ("io", lambda: L.pfe_step_io(h, N.vptr(fe), N.vptr(sats), 16, res))):
    fake.fake_clear_log()
    out[name] = [call(), launched("k_epoch"), launched("ObsInRing"), launched("ObsInline")]
""")
    assert r["step"] == r["per_filter"] == [0, 1, 1, 0] and r["io"] == [0, 1, 0, 1]


def test_velocities_with_nothing_to_follow_are_read_by_the_copy_engine(fake):
    """Nothing follows the read of an idle engine's control blocks, so it is a copy;
    the Doppler update's own kernels follow it."""
    r = run(fake, r"""
vs, v0, row = N.VelState(), np.zeros(3), np.zeros(1, N.DOPPLER_ROW_DTYPE)
vs.buf = block(2 * 12 * n * 8)
row["sat"], row["weight"] = 2e7, 1.0
N.check(L.pfe_vel_init(h, 0, C.byref(vs), N.dptr(v0), 0.1, 1.0, 0))
for name, call in (("follow", lambda: L.pfe_vel_follow(h, 0, C.byref(vs))),
                   ("doppler", lambda: L.pfe_vel_doppler(h, 0, C.byref(vs), N.vptr(row), 1, 0.19, 0.5, 0.0, 0.0, 0))):
    fake.fake_clear_log()
    out[name] = [call(), launched("k_mirror"), launched("k_doppler")]
""")
    assert r["follow"] == [0, 0, 0] and r["doppler"] == [0, 1, 1]
