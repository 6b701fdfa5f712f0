"""The two forms of the single-precision IMPLSCH, tiles of 32 sea points and a
warp per point, give the same bits.  Which one runs depends on the size of a
context's grid, so a grid and its pieces, each in a context of its own, may run
different forms: their integer decisions (JU, MIJ, LFACTOR's iterations, the
wind-sea masks) and spectra, TAUW, USTAR and Z0 must be equal all the same, and
latitude bands must reproduce the whole grid bit for bit whatever their size."""
import numpy as np
import pytest

from test_gpu_tile import _grid_case

pytestmark = pytest.mark.gpu


def _model(cfg, grid, depth):
    from wam_b200 import WamModel
    m = WamModel(cfg)
    m.set_grid(grid)
    m.set_depth(depth)
    m.prepare_propagation()
    m.prepare_source()
    return m


def _step(torch, m, f, fields):
    """One IMPLSCH on copies: spectrum, TAUW, USTAR, Z0, decisions, masks."""
    n, dev = f.shape[-1], f.device
    dec = torch.zeros((4, n), dtype=torch.int32, device=dev)
    ll = torch.zeros((2, f.shape[0], f.shape[1], n), dtype=torch.uint8, device=dev)
    m.set_diagnostics(dec, ll)
    x = [f.clone()] + [a.clone() for a in fields]
    torch.cuda.synchronize()
    m.implsch_dev(*x)
    m.sync()
    return [x[0], x[3], x[4], x[5], dec, ll]


# direction counts with and without a compiled instance, one to three directions per warp, a last
# warp that is not full, directions beyond 32 in one and in two warps, as few warps as the stress
# chain of SINPUT_ARD takes
@pytest.mark.parametrize("kl,ml,fr1,iphys,shallow,isnonlin", [
    (36, 30, 0.0345, 1, True, 0), (36, 30, 0.0345, 2, True, 0), (36, 35, 0.0345, 1, True, 1), (36, 25, 0.04177, 2, False, 0),
    (30, 29, 0.0345, 1, True, 0), (30, 29, 0.0345, 2, True, 1), (24, 25, 0.04177, 1, False, 0), (24, 25, 0.04177, 2, False, 0),
    (12, 25, 0.04177, 1, False, 0), (12, 25, 0.04177, 2, True, 0), (33, 30, 0.0345, 1, True, 0), (35, 25, 0.04177, 2, True, 0),
    (25, 26, 0.04177, 1, True, 1), (22, 25, 0.04177, 2, True, 0), (16, 25, 0.04177, 1, False, 0), (7, 25, 0.04177, 2, False, 0),
    (4, 25, 0.04177, 1, False, 0)])
def test_tiles_and_warps_agree_bit_for_bit(kl, ml, fr1, iphys, shallow, isnonlin):
    import torch
    from wam_b200 import regular_grid
    nx, ny, rows = 72, 75, 10
    w = _grid_case(kl, ml, fr1, iphys, shallow, isnonlin, nx, ny)
    dev = torch.device("cuda")
    t = lambda a: torch.tensor(np.asarray(a, np.float32), device=dev)
    whole = _model(w.cfg, w.grid, w.depth)
    assert whole.implsch_points() == 32
    pieces = []
    for r in range(0, ny, rows):
        k = min(rows, ny - r)
        g = regular_grid(np.ones((nx, k), bool), -20.0 + 0.8 * r, -60.0, 0.8, 0.8)
        lo, hi = nx * r, nx * (r + k)
        m = _model(w.cfg, g, w.depth[lo:hi])
        assert m.implsch_points() < 32
        pieces.append((m, lo, hi))
    f = w.spectrum_device(torch, dev)
    fields = [t(a) for a in (w.u10, w.udir, w.tauw, w.ustar, w.z0, w.roairn, w.wstar)]
    names = ("spectrum", "TAUW", "USTAR", "Z0", "decisions", "masks")
    for it in range(5):
        if it == 4:
            # bins too small for the quotients in single precision, and empty ones
            f[::3, ::2] *= 1e-30
            f[:, 1] = 0
        a = _step(torch, whole, f, fields)
        for m, lo, hi in pieces:
            b = _step(torch, m, f[:, :, lo:hi].contiguous(), [x[lo:hi].contiguous() for x in fields])
            for name, x, y in zip(names, a, b):
                assert torch.equal(x[..., lo:hi], y), (it, lo, name, int((x[..., lo:hi] != y).sum()))
        f, fields = a[0], fields[:2] + a[1:4] + fields[5:]
    whole.close()
    for m, _, _ in pieces:
        m.close()


@pytest.mark.parametrize("name,scale,nbands", [("c1", 0.1, 8), ("c2", 0.2, 3)])
def test_bands_below_the_tile_size_match_whole_grid(name, scale, nbands):
    """As test_gpu_bands, on a grid that runs on tiles whose bands do not."""
    import torch
    from wam_b200 import WamModel
    from wam_b200.halo import exchange_plan, local_grid, partition
    from wam_b200.synth import make_workload
    w = make_workload(name, scale=scale)
    dev = torch.device("cuda", 0)
    nprop = w.cfg["idelt"] // w.cfg["idelpro"]
    t = lambda a: torch.tensor(np.asarray(a, np.float32), device=dev)
    g = _model(w.cfg, w.grid, w.depth)
    F = w.spectrum_device(torch, dev)
    S = torch.empty_like(F)
    G = [t(a) for a in (w.u10, w.udir, w.tauw, w.ustar, w.z0, w.roairn, w.wstar)]
    parts = partition(w.grid, nbands)
    bands = []
    for p in parts:
        cut = slice(p["ninf"], p["nsup"])
        m = WamModel(w.cfg)
        m.set_grid(local_grid(w.grid, p))
        m.set_depth(np.asarray(w.depth)[cut])
        m.set_owned(p["lo"] - p["ninf"], p["hi"] - p["ninf"])
        m.prepare_propagation()
        m.set_counter(g.counter)
        m.prepare_source()
        bands.append([m, p, F[:, :, cut].clone(), [x[cut].clone() for x in G]])
    assert g.implsch_points() == 32 and all(b[0].implsch_points() < 32 for b in bands)
    for step in range(3):
        g.step_dev(F, nprop, *G, scratch=S)
        g.sync()
        src, dst = [b[2] for b in bands], [torch.empty_like(b[2]) for b in bands]
        for _ in range(nprop * g.counter):
            for r, (_, p, _, _) in enumerate(bands):
                for q, lo, hi in exchange_plan(parts, r)[1]:
                    o = parts[q]["ninf"]
                    src[r][:, :, lo - p["ninf"]:hi - p["ninf"]] = src[q][:, :, lo - o:hi - o]
            torch.cuda.synchronize()
            for r, b in enumerate(bands):
                b[0].propags_substep_dev(src[r], dst[r])
                b[0].sync()
            src, dst = dst, src
        for r, b in enumerate(bands):
            b[0].implsch_dev(src[r], *b[3])
            b[0].sync()
            b[2], p = src[r], b[1]
            own, all_ = slice(p["lo"] - p["ninf"], p["hi"] - p["ninf"]), slice(p["lo"], p["hi"])
            assert torch.equal(b[2][:, :, own], F[:, :, all_]), f"step {step} band {r} spectrum"
            for i in (2, 3, 4):
                assert torch.equal(b[3][i][own], G[i][all_]), f"step {step} band {r} field {i}"
    g.close()
    for b in bands:
        b[0].close()
