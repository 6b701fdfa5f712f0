"""PROPAGS with currents, two frequencies per thread: COUNTER > 1 (every
coefficient divided), odd and even frequency counts, the smallest spectra, and
the batched launch.  Bit-exact against the oracle or the member's own step."""
import numpy as np
import pytest

from test_gpu_propags_variants import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("idelpro", [600, 7200])
@pytest.mark.parametrize("ml", [24, 25])
@pytest.mark.parametrize("spherical,shallow,reduced", [(0, 0, 0), (0, 1, 0), (1, 0, 0), (1, 1, 0), (1, 0, 1), (1, 1, 1)])
def test_currents_counter_and_frequencies(oracle_mod, spherical, shallow, reduced, ml, idelpro):
    from wam_b200 import WamModel
    cfg, g, depth, u, v, f = _case(oracle_mod, spherical, shallow, 1, reduced, shallow, idelpro=idelpro)
    cfg = dict(cfg, ml=ml)
    f = np.asfortranarray(f[:, :, :ml])
    o = oracle_mod.Oracle(cfg)
    o.set_grid(g)
    o.set_fields(depth, u, v)
    rc, cfl, cnt = o.prepare_propagation()
    m = WamModel(cfg)
    m.set_grid(g)
    m.set_depth(depth)
    m.set_current(u, v)
    if rc != 0:
        with pytest.raises(Exception):
            m.prepare_propagation()
        return
    gcfl, gcnt = m.prepare_propagation()
    assert gcnt == cnt and np.float32(gcfl) == np.float32(cfl)
    assert cnt > 1 or idelpro == 600
    ref = o.propags(f.astype(float)).astype(np.float32)
    got = f.copy(order="F")
    m.propags(got)
    assert np.array_equal(got, ref), float(np.abs(got - ref).max())
    m.close()


@pytest.mark.parametrize("spherical,shallow", [(1, 0), (1, 1)])
def test_currents_batched(oracle_mod, spherical, shallow):
    import torch
    from wam_b200 import WamModel
    from wam_b200.batch import WamBatch
    models, ref, bat = [], [], []
    for seed in (3, 4):
        cfg, g, depth, u, v, f = _case(oracle_mod, spherical, shallow, 1, 0, shallow, seed=seed)
        m = WamModel(cfg)
        m.set_grid(g)
        m.set_depth(depth)
        m.set_current(u, v)
        m.prepare_propagation()
        m.prepare_source()
        n = g["nsea"]
        t = lambda a: torch.full((n,), a, dtype=torch.float32, device="cuda")
        st = [torch.tensor(np.ascontiguousarray(f.transpose(2, 1, 0)), device="cuda") * 0.01]
        st += [torch.zeros_like(st[0])] + [t(a) for a in (9.0, 0.7, 0.05, 0.0, 0.0, 1.22, 0.0)]
        models.append(m)
        ref.append(st)
        bat.append([x.clone() for x in st])
    torch.cuda.synchronize()
    b = WamBatch(models)
    for k, st in enumerate(bat):
        b.set_member(k, *st)
    b.step()
    b.sync()
    torch.cuda.synchronize()
    for m, st in zip(models, ref):
        fl, sc, u10, udir, tauw, ustar, z0, roairn, wstar = st
        m.step_dev(fl, 1, u10, udir, tauw, ustar, z0, roairn, wstar, scratch=sc)
        m.sync()
    for a, c in zip(ref, bat):
        assert torch.equal(a[0], c[0]) and torch.equal(a[4], c[4])
    b.close()
    for m in models:
        m.close()
