"""The step on host arrays cut into many chunks (a chunk has at least a quarter of
the SMs' tiles, so that takes a large grid), IMPLSCH of consecutive chunks on four
streams: bit for bit the step on device arrays, over two passes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,scale", [("c1", 0.33), ("c2", 0.7)])
def test_many_chunks_equal_device_step(name, scale):
    import torch
    from wam_b200 import WamModel
    from wam_b200.synth import make_workload
    w = make_workload(name, scale=scale)
    assert w.nsea > 40000
    m = WamModel(w.cfg)
    m.set_grid(w.grid)
    m.set_depth(w.depth)
    m.prepare_propagation()
    m.prepare_source()
    dev = torch.device("cuda", 0)
    t = lambda a: torch.tensor(np.asarray(a, np.float32), device=dev)
    f = w.spectrum_device(torch, dev)
    s = torch.empty_like(f)
    D = [t(a) for a in (w.u10, w.udir, w.tauw, w.ustar, w.z0, w.roairn, w.wstar)]
    h = f.cpu().numpy().copy()
    H = [x.cpu().numpy().copy() for x in D]
    nprop = w.cfg["idelt"] // w.cfg["idelpro"]
    for step in range(2):
        m.step_dev(f, nprop, *D, scratch=s)
        m.sync()
        m.step(h, nprop, *H)
        assert np.array_equal(f.cpu().numpy(), h), step
        for i in (2, 3, 4):
            assert np.array_equal(D[i].cpu().numpy(), H[i]), (step, i)
    m.close()
