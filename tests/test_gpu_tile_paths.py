"""Where IMPLSCH runs on tiles: the size of grid from which it does, and the
calls that reach the tiles in other ways than a plain step, a batched ensemble
(directly and from its captured graph) and a checkpointed ST6 step, whose adjoint
takes the RTAU that the tiles recorded."""
import numpy as np
import pytest

from test_gpu_batch import _model, _state
from test_gpu_tile import _grid_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kl,ml,fr1,iphys,shallow", [(24, 25, 0.04177, 1, False), (24, 25, 0.04177, 2, False),
                                                     (36, 30, 0.0345, 1, True), (36, 30, 0.0345, 2, True)])
def test_tiles_from_the_first_point_beyond_a_wave(kl, ml, fr1, iphys, shallow):
    """144 to 148 registers a thread leave 12 warps on an SM whatever shared
    memory would hold: 1776 points are one wave of the warp-per-point form."""
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the sizes are those of 148 SMs")
    for nx, ny, tile in ((48, 37, False), (53, 34, True), (60, 50, True)):
        w = _grid_case(kl, ml, fr1, iphys, shallow, 0, nx, ny)
        m = _model(w)
        assert (m.implsch_points() == 32) == tile, (nx * ny, m.implsch_points())
        m.close()


def test_batch_on_tiles_matches_members():
    import torch
    from wam_b200.batch import WamBatch
    from wam_b200.synth import make_ensemble, make_workload
    dev = torch.device("cuda", 0)
    ws = make_ensemble(n_members=5, seed=31, size_range=(2000, 9000)) + [make_workload("c1", scale=0.05), make_workload("c1", scale=0.02)]
    models = [_model(w) for w in ws]
    on = [m.implsch_points() == 32 for m in models]
    assert sum(on) >= 4 and not all(on)
    assert {w.cfg["iphys"] for w, t in zip(ws, on) if t} == {1, 2}
    ref = [_state(torch, w, dev) for w in ws]
    bat = [[x.clone() for x in st] for st in ref]
    torch.cuda.synchronize()
    b = WamBatch(models)
    for g, st in enumerate(bat):
        b.set_member(g, *st)
    for it in range(4):
        if it == 2:
            b.capture()
        for w, m, (f, sc, *rest) in zip(ws, models, ref):
            m.step_dev(f, w.cfg["idelt"] // w.cfg["idelpro"], *rest, scratch=sc)
            m.sync()
        b.step()
        b.sync()
        for g, (a, c) in enumerate(zip(ref, bat)):
            for i in (0, 4, 5, 6):
                assert torch.equal(a[i], c[i]), f"pass {it} member {g} field {i}"
    b.close()
    for m in models:
        m.close()


@pytest.mark.parametrize("kl,ml,fr1,shallow", [(36, 30, 0.0345, True), (24, 25, 0.04177, False)])
def test_st6_checkpoint_of_a_tile_step(kl, ml, fr1, shallow):
    """Two checkpointed source steps and their adjoints on a grid that runs on
    tiles, against its pieces, which run on warps: gradients bit for bit."""
    import torch
    from wam_b200 import WamModel, regular_grid
    nx, ny, rows = 72, 75, 15
    w = _grid_case(kl, ml, fr1, 2, shallow, 0, nx, ny)
    dev = torch.device("cuda")
    t = lambda a: torch.tensor(np.asarray(a, np.float32), device=dev)
    F = w.spectrum_device(torch, dev)
    U, D, R, W = (t(a) for a in (w.u10, w.udir, w.roairn, w.wstar))
    g = torch.Generator(device=dev).manual_seed(4)
    lam = torch.randn(F.shape, generator=g, device=dev)

    def window(grid, depth, lo, hi):
        m = WamModel(w.cfg)
        m.set_grid(grid)
        m.set_depth(depth)
        m.prepare_propagation()
        m.prepare_source()
        c = lambda x: x[..., lo:hi].contiguous().clone()
        f, lf, u, d, r, ws = (c(x) for x in (F, lam, U, D, R, W))
        tw, us, z0, lt = (torch.zeros(hi - lo, device=dev) for _ in range(4))
        lu = [torch.empty_like(u) for _ in range(2)]
        sc = torch.empty_like(f)
        m.checkpoint_reserve(2, hi - lo)
        torch.cuda.synchronize()
        for p in range(2):
            m.step_ckpt_dev(p, f, 0, u, d, tw, us, z0, r, ws, scratch=sc)
        for p in (1, 0):
            m.step_adj_dev(p, 0, lf, lt, lu[p], d, r, ws, scratch=sc)
        m.sync()
        n = m.implsch_points()
        m.close()
        return n, [f, tw, lf, lt] + lu

    n, whole = window(w.grid, w.depth, 0, nx * ny)
    assert n == 32
    assert all(torch.isfinite(x).all() for x in whole) and float(whole[2].abs().max()) > 0
    for r in range(0, ny, rows):
        lo, hi = nx * r, nx * (r + rows)
        n, piece = window(regular_grid(np.ones((nx, rows), bool), -20.0 + 0.8 * r, -60.0, 0.8, 0.8), w.depth[lo:hi], lo, hi)
        assert n < 32
        for q, (a, b) in enumerate(zip(whole, piece)):
            assert torch.equal(a[..., lo:hi], b), (lo, q)
