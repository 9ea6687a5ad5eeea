"""Orbits of a few satellites over long series: the edges of their tiles of 256 and
1024 epochs against the oracle (the check and its tolerance are those of
tests/test_orbit_tiles_gpu.py), and the time: one satellite takes less than half of
what eight take (a quarter is usual; with tiles of eight satellites it took the
same)."""
import numpy as np
import pytest

from test_orbit_tiles_gpu import test_orbits_match_oracle_at_tile_edges as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne,ns,step", [(255, 1, 60.0), (257, 2, 59.3), (1023, 3, 60.0), (1025, 4, 60.0), (300, 5, 60.0),
                                        (606_209, 1, 60.0), (151_553, 4, 60.0)])
def test_few_satellites_match_oracle_at_tile_edges(ne, ns, step):
    _check(ne, ns, step)


def test_one_satellite_costs_less_than_eight():
    import torch
    from gnss_gpu_b200 import _native as N
    L, ne = N.load(), 1_000_000
    t = torch.linspace(0.0, 7200.0, ne, dtype=torch.float64, device="cuda")

    def times(ns):
        rec = np.zeros(ns, N.BROADCAST_DTYPE)
        rec["system"] = ord("G")
        rec["kepler"]["sqrt_a"], rec["kepler"]["e"], rec["kepler"]["M0"] = 5153.7, 0.01, np.arange(ns)
        d = torch.from_numpy(rec.view(np.uint8).copy()).cuda()
        pos = torch.empty((ne, ns, 3), dtype=torch.float64, device="cuda")
        clk = torch.empty((ne, ns), dtype=torch.float64, device="cuda")
        out = []
        for _ in range(15):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            N.check(L.pf_broadcast_orbits(d.data_ptr(), ns, None, t.data_ptr(), ne, ns, 60.0, pos.data_ptr(),
                                          clk.data_ptr(), torch.cuda.current_stream().cuda_stream))
            b.record()
            torch.cuda.synchronize()
            out.append(a.elapsed_time(b))
        return np.median(out[3:])

    assert times(1) < 0.5 * times(8)
