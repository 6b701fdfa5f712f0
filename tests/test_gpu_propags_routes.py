"""A PROPAGS sub-step takes one or two frequencies per thread, by precision,
variant, COUNTER and the size of the launch.  The bits do not depend on it: a
sub-step of the whole grid (two frequencies where they pay) against the same
sub-step in ranges of 128 points (a launch of few CTAs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [4, 8])
@pytest.mark.parametrize("idelpro", [300, 3600])
@pytest.mark.parametrize("kl,ml,shallow,refr_d,currents", [(36, 30, True, True, False), (36, 29, True, False, False),
                                                           (24, 25, False, False, False), (36, 30, True, True, True),
                                                           (24, 25, False, False, True)])
def test_whole_launch_equals_small_ranges(kl, ml, shallow, refr_d, currents, idelpro, precision):
    import torch
    from wam_b200 import WamModel, make_config, regular_grid
    nx, ny = 67, 50
    rng = np.random.default_rng(kl + ml)
    sea = rng.random((nx, ny)) > 0.05
    g = regular_grid(sea, -30.0, -60.0, 0.4, 0.4)
    n = g["nsea"]
    cfg = make_config(kl, ml, 0.0345, 2, 3600, idelpro, g["delphi"], shallow_run=shallow, refraction_d_run=refr_d,
                      refraction_c_run=currents, precision=precision)
    m = WamModel(cfg)
    m.set_grid(g)
    m.set_depth(rng.uniform(20.0, 300.0, n).astype(np.float32) if shallow else np.full(n, 4000.0, np.float32))
    if currents:
        m.set_current(rng.uniform(-0.3, 0.3, n).astype(np.float32), rng.uniform(-0.3, 0.3, n).astype(np.float32))
    m.prepare_propagation()
    assert (m.counter > 1) == (idelpro == 3600)
    dt = torch.float32 if precision == 4 else torch.float64
    f = torch.tensor(rng.random((ml, kl, n)), dtype=dt, device="cuda")
    a, b = torch.full_like(f, -1.0), torch.full_like(f, -2.0)
    torch.cuda.synchronize()
    m.propags_substep_dev(f, a)
    for lo in range(0, n, 128):
        m.propags_substep_range_dev(f, b, lo, min(lo + 128, n))
    m.sync()
    assert torch.equal(a, b), int((a != b).sum())
    m.close()


@pytest.mark.parametrize("idelpro", [3600, 14400])
@pytest.mark.parametrize("spherical,shallow,reduced,refr_d", [(0, 0, 0, 0), (0, 1, 0, 1), (1, 0, 0, 0), (1, 0, 1, 0), (1, 1, 0, 0),
                                                              (1, 1, 1, 1)])
def test_quotients_by_counter_match_the_oracle(oracle_mod, spherical, shallow, reduced, refr_d, idelpro):
    """Without currents every coefficient is divided by COUNTER as a scaled
    quotient of its own: bit for bit the oracle's division."""
    from test_gpu_propags_variants import _case
    from wam_b200 import WamModel
    cfg, g, depth, _, _, f = _case(oracle_mod, spherical, shallow, 0, reduced, refr_d, idelpro=idelpro)
    o = oracle_mod.Oracle(cfg)
    o.set_grid(g)
    o.set_fields(depth)
    rc, _, cnt = o.prepare_propagation()
    assert rc == 0 and cnt > 1
    m = WamModel(cfg)
    m.set_grid(g)
    m.set_depth(depth)
    m.prepare_propagation()
    ref = o.propags(f.astype(float)).astype(np.float32)
    got = f.copy(order="F")
    m.propags(got)
    assert np.array_equal(got, ref), float(np.abs(got - ref).max())
    m.close()
