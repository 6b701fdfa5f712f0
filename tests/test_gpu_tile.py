"""IMPLSCH on tiles of 32 sea points (grids of more points than the warp-per-point
kernel holds at once) against the FP32 oracle: integer decisions and spectra on
a sample of the points, for direction counts with and without a compiled
instance (even and odd, a last column group that is not full), tiles that end
past the last point, both physics, depth and deep runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid_case(kl, ml, fr1, iphys, shallow, isnonlin, nx=61, ny=47):
    """An open ocean of 2867 points (89 full tiles and one of 19) with winds,
    depths and peak frequencies that vary over it."""
    from wam_b200 import make_config, regular_grid
    from wam_b200.synth import Workload, grf, jonswap_factors, _unit
    rng = np.random.default_rng(kl * 100 + iphys)
    sea = np.ones((nx, ny), bool)
    g = regular_grid(sea, -20.0, -60.0, 0.8, 0.8)
    cfg = make_config(kl, ml, fr1, iphys, 600, 120, g["delphi"], shallow_run=shallow, refraction_d_run=shallow,
                      isnonlin=isnonlin, betamax=1.42 if iphys == 1 else 1.20)
    pick = lambda a: a.T.ravel().astype(np.float32)
    depth = pick(12.0 * 300.0 ** _unit(grf(rng, nx, ny, 6))) if shallow else np.full(nx * ny, 4000.0, np.float32)
    u10 = pick(3.0 + 20.0 * _unit(grf(rng, nx, ny, 5)))
    udir = pick(2 * np.pi * _unit(grf(rng, nx, ny, 8)))
    fr = fr1 * 1.1 ** np.arange(ml)
    th = (np.arange(kl) + 0.5) * (2 * np.pi / kl)
    fp = 0.07 + 0.18 * pick(_unit(grf(rng, nx, ny, 5)))
    e, d = jonswap_factors(fr, th, fp, 0.018, 3.3, 0.07, 0.09, udir)
    w = Workload("tile", cfg, g, depth, u10, udir, e, d)
    w.wstar = rng.uniform(0.0, 1.2, w.nsea).astype(np.float32)
    return w


@pytest.mark.parametrize("kl,ml,fr1,iphys,shallow,isnonlin", [
    (36, 30, 0.0345, 1, True, 0), (36, 30, 0.0345, 2, True, 0), (24, 25, 0.04177, 1, False, 0),
    (24, 25, 0.04177, 2, False, 0), (36, 35, 0.0345, 1, True, 0), (30, 29, 0.0345, 2, True, 1),
    (12, 25, 0.04177, 2, True, 0), (25, 26, 0.04177, 1, True, 1), (35, 25, 0.04177, 2, True, 0),
    (16, 25, 0.04177, 1, False, 0), (7, 25, 0.04177, 2, False, 0)])
def test_tile_step_matches_oracle(oracle_mod, kl, ml, fr1, iphys, shallow, isnonlin):
    from wam_b200 import WamModel
    w = _grid_case(kl, ml, fr1, iphys, shallow, isnonlin)
    m = WamModel(w.cfg)
    m.set_grid(w.grid)
    m.set_depth(w.depth)
    m.prepare_propagation()
    m.prepare_source()
    o = oracle_mod.Oracle(w.cfg)
    o.set_grid(w.grid)
    o.set_fields(w.depth)
    o.prepare_propagation()
    o.prepare_source()
    # an evolved sea state: one step of the oracle first
    z = np.zeros(w.nsea)
    f, tw, us, zz, _ = o.implsch(w.spectrum_f().astype(float), w.u10, w.udir, z, z, z, w.roairn, w.wstar, w.depth,
                                 o.indep())
    f, tw = np.asfortranarray(f, np.float32), tw.astype(np.float32)
    fo, two, uso, zo, _, od = o.implsch_diag(f.astype(float), w.u10, w.udir, tw, us, zz, w.roairn, w.wstar, w.depth,
                                             o.indep())
    fg, tg, ug, zg = f.copy(order="F"), tw.copy(), np.zeros(w.nsea, np.float32), np.zeros(w.nsea, np.float32)
    gd = m.implsch_decisions(fg, w.u10, w.udir, tg, ug, zg, w.roairn, w.wstar)
    # at most 0.5 % of the points may decide otherwise, at a rounding boundary
    flip = np.zeros(w.nsea, bool)
    for q in ("JU", "MIJ1", "MIJ2", "LFIT"):
        flip |= gd[q] != od[q]
    for q in ("LLWS1", "LLWS2"):
        flip |= (gd[q] != od[q]).any(axis=(1, 2))
    assert flip.mean() <= 0.005, flip.sum()
    # one FP32 step: 1e-5 of the point's largest bin, as the parity tests
    err = np.abs(fg - fo).max(axis=(1, 2)) / fo.max(axis=(1, 2))
    assert err[~flip].max() <= 1e-5
    assert (np.abs(ug - uso) / uso)[~flip].max() <= 1e-5
    assert (np.abs(tg - two) / np.maximum(np.abs(two), 1e-3 * np.abs(two).max()))[~flip].max() <= 1e-5
    m.close()
