"""Integrated output over owned ranges that end inside a tile of 32 sea points.

Every point's parameters are a function of that point alone, so a range gives
the same bits as the whole grid (itself checked against the oracle in
test_gpu_output.py), writes 0 to the parameters it does not compute and leaves
the points outside the range as they were."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SWELL = [17, 18, 19, 20, 21, 22, 23, 25, 26, 27, 28, 29, 30, 31]
OWN = [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 32, 40]


@pytest.mark.parametrize("precision", [4, 8])
@pytest.mark.parametrize("name,scale", [("c0", 0.3), ("c1", 0.02)])
@pytest.mark.parametrize("i0,n", [(0, 1), (5, 31), (1, 32), (7, 33), (3, 97)])
def test_output_ranges(name, scale, i0, n, precision):
    import torch
    from wam_b200 import WamModel
    from wam_b200.synth import make_workload, vary_sea_state
    w = vary_sea_state(make_workload(name, scale=scale))
    dt = torch.float64 if precision == 8 else torch.float32
    t = lambda a: torch.tensor(np.asarray(a), dtype=dt, device="cuda")
    f = t(np.ascontiguousarray(np.asarray(w.spectrum_f()).transpose(2, 1, 0)))
    us = 0.04 * t(w.u10)
    z0 = us * us * 0.0012
    got = []
    for lo, hi in ((0, w.nsea), (i0, i0 + n)):
        m = WamModel(dict(w.cfg, precision=precision))
        m.set_grid(w.grid)
        m.set_depth(w.depth)
        m.set_owned(lo, hi)
        m.prepare_propagation()
        m.prepare_source()
        blk = torch.full((40, w.nsea), 7.0, dtype=dt, device="cuda")
        u10, udir, tauw, us0, z00 = t(w.u10), t(w.udir), t(w.tauw), us.clone(), z0.clone()
        torch.cuda.synchronize()  # the model's stream is its own
        m.output_parameters_dev(f, u10, udir, tauw, us0, z00, block=blk)
        m.sync()
        first = blk.clone()
        torch.cuda.synchronize()
        m.output_swell_dev(f, udir, us, blk)
        m.sync()
        got.append((first.cpu().numpy(), blk.cpu().numpy()))
        m.close()
    inside = np.zeros(w.nsea, bool)
    inside[i0:i0 + n] = True
    for whole, part in zip(got[0], got[1]):
        assert np.array_equal(part[:, inside], whole[:, inside])
        assert np.all(part[:, ~inside] == 7.0)
    rest = [p - 1 for p in range(1, 41) if p not in OWN]
    assert np.all(got[1][0][rest][:, inside] == 0)
    assert np.all(got[1][1][[p - 1 for p in (24, 33, 39)]][:, inside] == 0)
    assert np.all(got[1][1][[p - 1 for p in SWELL]][:, inside] != 7.0)
