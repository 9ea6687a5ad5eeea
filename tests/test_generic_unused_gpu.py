"""A satellite of weight 0 in the device filter's likelihoods adds nothing,
whatever its record holds: pseudoranges beyond FP32 and a position at the
receiver give the log-weights of the set without it, bit for bit (the remaining
satellites are added in the same order)."""
import numpy as np
import pytest

from conftest import TOKYO_PR, TOKYO_SATS, TOKYO_TRUE_CB, TOKYO_TRUE_POS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gate", [0.0, 30.0])
@pytest.mark.parametrize("kind", ["gaussian", "huber", "student_t", "gmm"])
def test_weight_zero_records_are_skipped(kind, gate):
    from gnss_gpu_b200 import _native as N
    from gnss_gpu_b200.engine import Engine, EngineOptions, FilterSpec
    eng = Engine([FilterSpec(n_particles=1003, seed=3)], EngineOptions(n_clk=1, weight_mode="generic", max_sats=16))
    eng.set_likelihood(kind, nu=4.0, gate_m=gate)
    fl = N.PF_EP_WEIGHT | N.PF_EP_NO_RESAMPLE

    def log_weights(sats, pr, w):
        eng.initialize(0, TOKYO_TRUE_POS, TOKYO_TRUE_CB, 5.0, 3.0)
        fe, sv = eng.pack_epoch([dict(sats=sats, pr=pr, w=w, flags=fl)])
        eng.step_io(fe, sv)
        return eng.state_f32(0)[1]

    ns = len(TOKYO_SATS)
    want = log_weights(TOKYO_SATS, TOKYO_PR, np.ones(ns))
    at = [0, 2, 2, ns]
    sats = np.insert(TOKYO_SATS, at, TOKYO_SATS[0], axis=0)
    pr = np.insert(TOKYO_PR, at, [1.7e308, -1e300, 1e39, 0.0])
    w = np.insert(np.ones(ns), at, 0.0)
    sats[-1] = TOKYO_TRUE_POS
    got = log_weights(sats, pr, w)
    assert np.all(np.isfinite(want))
    np.testing.assert_array_equal(got, want)
