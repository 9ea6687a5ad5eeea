"""What a call takes to the GPU and back without the copy engine: observation rows
as a kernel parameter (one size up to 32 rows, a larger one up to 128) against the
FP64 oracle, and the control blocks' mirror written by a kernel (up to 8 KB of
blocks, about 16 filters; more go by a copy) against the results of the one-call
step, which are written by the epoch kernel: the same bytes."""
import numpy as np
import pytest

from oracle import oracle as O
from test_obs_term_sizes_gpu import test_obs_term_matches_oracle_at_edges as _check_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [O.OBS_DD_PSEUDORANGE, O.OBS_CARRIER_AFV, O.OBS_DD_CARRIER_AFV])
@pytest.mark.parametrize("rows", [31, 32, 33])
def test_rows_at_the_edge_of_the_small_parameter(kind, rows):
    _check_rows(kind, 300, rows, 0.2, 1.0, 2)


@pytest.mark.parametrize("n_filters", [1, 2, 14, 15, 16, 17, 18, 40])
def test_read_results_equal_the_one_call_step(n_filters):
    from gnss_gpu_b200.engine import Engine, EngineOptions, FilterSpec
    rng = np.random.default_rng(n_filters)
    p0 = np.array([-3957199.0, 3310205.0, 3737911.0])
    sats = p0 + 2.1e7 * (lambda d: d / np.linalg.norm(d, axis=1, keepdims=True))(rng.normal(size=(6, 3)))
    pr = np.linalg.norm(sats - p0, axis=1) + 30.0 + rng.normal(0, 2.0, 6)
    outs = []
    for one_call in (True, False):
        eng = Engine([FilterSpec(n_particles=50 + 3 * f, seed=f) for f in range(n_filters)],
                     EngineOptions(n_clk=1, max_sats=8))
        for f in range(n_filters):
            eng.initialize(f, p0, 30.0, 20.0, 5.0)
        for _ in range(3):
            fe, rec = eng.pack_epoch([dict(sats=sats, pr=pr)] * n_filters)
            if one_call:
                r = eng.step_io(fe, rec)
            else:
                eng.upload(0, fe, rec)
                eng.step()
                r = eng.results_array()
        outs.append(bytes(r))
    assert outs[0] == outs[1]
