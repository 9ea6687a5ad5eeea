"""A device error of an earlier step (here a bounded wait that runs out) is reported
by the next observation term, which then leaves the log-weights as they are: the
same bytes as without the call."""
import numpy as np
import pytest

from gnss_gpu_b200 import _native as N
from oracle import oracle as O

import pfhelp as H
from conftest import TOKYO_PR, TOKYO_SATS, TOKYO_TRUE_CB, TOKYO_TRUE_POS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("kind", [O.OBS_DD_PSEUDORANGE, O.OBS_CARRIER_AFV, O.OBS_DD_CARRIER_AFV])
def test_observation_term_after_a_device_error(kind, accumulate):
    rows = np.zeros(4, N.OBS_ROW_DTYPE)
    rows["sat_k"], rows["sat_ref"], rows["weight"], rows["wavelength"] = TOKYO_SATS[1:5], TOKYO_SATS[0], 1.0, 0.19

    def log_weights(with_term):
        eng = H.make_engine([3001], seeds=[5])
        eng.initialize(0, TOKYO_TRUE_POS, TOKYO_TRUE_CB, 5.0, 3.0)
        fe, sv = eng.pack_epoch([dict(sats=TOKYO_SATS, pr=TOKYO_PR, flags=N.PF_EP_WEIGHT | N.PF_EP_NO_RESAMPLE)])
        eng.set_spin_limit(2000)
        eng.poison_lookback(True)
        eng.upload(0, fe, sv)
        eng.step()
        assert eng.error_word() != 0
        if with_term:
            with pytest.raises(N.PFError) as ei:
                eng.add_obs_term(0, kind, rows, 1.0, accumulate=accumulate)
            assert ei.value.status == N.PF_ETIMEOUT
        eng.poison_lookback(False)  # clears the error word
        eng.set_spin_limit(0)
        lw = eng.state_f32(0, raw=True)[1].copy()
        eng.close()
        return lw

    want = log_weights(False)
    assert np.ptp(want) > 0.0
    np.testing.assert_array_equal(log_weights(True), want)
