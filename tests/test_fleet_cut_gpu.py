"""A fleet's tiles on the CTAs, cut by cost or by number: on both sides of the rule (on
average eight tiles of 1024 particles per filter, more tiles than CTAs) a step gives
every filter the bytes that a launch of its own gives it, and many small filters take
less than the chain of kernels (three quarters is usual; with the cut by cost they
took more)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N_SAT = 12


def _fleet(counts, sats_of, **opt):
    from gnss_gpu_b200 import _native as N
    from gnss_gpu_b200.engine import Engine, EngineOptions, FilterSpec
    rng = np.random.default_rng(len(counts))
    p0 = np.array([-3957199.0, 3310205.0, 3737911.0])
    up, flags = p0 / np.linalg.norm(p0), N.PF_EP_PREDICT | N.PF_EP_WEIGHT | opt.pop("flags", 0)
    eng = Engine([FilterSpec(n_particles=int(n), seed=11 + k) for k, n in enumerate(counts)],
                 EngineOptions(n_clk=1, max_sats=N_SAT, weight_mode="huber", **opt))
    epochs = []
    for k in range(len(counts)):
        eng.initialize(k, p0, 100.0, 5.0, 5.0)
        u = rng.normal(size=(sats_of(k), 3)) + 2.0 * up
        sats = p0 + 2.2e7 * u / np.linalg.norm(u, axis=1)[:, None]
        pr = np.linalg.norm(sats - p0, axis=1) + 100.0 + rng.normal(0, 3, len(sats))
        epochs.append(dict(disp=np.zeros(3), sats=sats, pr=pr, w=np.ones(len(sats)), flags=flags))
    eng.upload(0, *eng.pack_epoch(epochs))
    return eng


@pytest.mark.parametrize("counts", [[7 * 1024 + 1000] * 41 + [7 * 1024], [7 * 1024 + 1] * 41, [8 * 1024] * 40,
                                    [1] * 22 + [15 * 1024 + 1] * 21 + [9 * 1024],
                                    [300] * 30 + [20_000, 1023, 150_001, 1025] * 6])
def test_same_bytes_as_a_launch_per_filter(counts):
    sats_of = lambda k: 4 + (5 * k) % (N_SAT - 3)  # noqa: E731
    one, many = _fleet(counts, sats_of), _fleet(counts, sats_of)
    for _ in range(3):
        many.step()
        one.step_per_filter()
    assert many.results_array().tobytes() == one.results_array().tobytes()
    for k in (0, len(counts) // 2, len(counts) - 1):
        a, b = many.state_f32(k), one.state_f32(k)
        for x, y in zip(a, b):
            assert np.asarray(x).tobytes() == np.asarray(y).tobytes()


def test_many_small_filters_cost_less_than_the_chain():
    from gnss_gpu_b200 import _native as N

    def kernel_time(chain):
        eng = _fleet([300] * 4096, lambda k: 8, kernel_chain=chain, flags=N.PF_EP_NO_RESAMPLE)
        out = []
        for _ in range(15):
            eng.synchronize()
            t = time.perf_counter()
            for _ in range(10):
                eng.step()
            eng.synchronize()
            out.append(time.perf_counter() - t)
        return np.median(out[3:])

    assert kernel_time(False) < 0.92 * kernel_time(True)
