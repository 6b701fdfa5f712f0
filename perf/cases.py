"""Timed cases of the wave-model library: what a user's program has it do.

Each case is one call (or one pass of calls) through the public entry points
of `wam_b200`: whole source steps, the two kernels of a step by themselves, a
batched ensemble, an assimilation window with its adjoint, the integrated
output and the drop-in step on host arrays.  `listed()` gives the fixed cases,
`draw()` more of the same ranges.  Grids, winds and sea states are synthetic
and made from the seed alone; the recipes (grid sizes, spectral grids, time
steps, depth ranges) are those of the repository's own workloads.

`exact()` evaluates the same model equations in float64 with plain torch and
numpy.
"""
import functools
import math

import numpy as np
import torch

from wam_b200 import WamModel, make_config
from wam_b200.batch import WamBatch

DEV = "cuda"
G, PI = 9.806, 3.1415927
ZPI, RAD_E = 2.0 * PI, 40000000.0 / (2.0 * PI)
CIRC = 40000000.0
NDEPTH, DEPTHA, DEPTHD = 69, 1.0, 1.1


# ---------------------------------------------------------------- the cases

def _case(kind, nx, ny, **kw):
    c = dict(kind=kind, nx=nx, ny=ny, lat0=-45.0, lon0=-60.0, dlat=0.3, dlon=0.3, land=0.3, kl=36, ml=30, fr1=0.0345,
             iphys=2, shallow=True, refr_d=True, refr_c=False, idelt=600, idelpro=120, dmin=10.0, dmax=5000.0,
             gust=0.0, pad=0, f64=False, isnonlin=0, members=0, passes=0)
    c.update(kw)
    return c


def listed():
    deep = dict(lat0=20.0, lon0=-40.0, land=0.1, kl=24, ml=25, fr1=0.04177, shallow=False, refr_d=False, idelt=900,
                idelpro=900, dmin=4000.0, dmax=4000.0)
    return [
        # a harbour-sized nest: a few warps of work, launches and latency count
        _case("step", 15, 10, name="coastal_step_st4", iphys=1, **dict(deep, dlat=1.0, dlon=1.0)),
        # the FP64 reference run that FP32 results are checked against
        _case("implsch", 72, 50, name="reference_implsch_fp64", dlat=1.0, dlon=1.0, f64=True),
        # the source terms alone, ST6 physics, a regional grid with an odd leading dimension
        _case("implsch", 600, 450, name="regional_implsch_st6", dlat=0.2, dlon=0.2, pad=3),
        # the source terms alone, ST4 physics with gustiness, the assimilation grid
        _case("implsch", 400, 300, name="shelf_implsch_st4", iphys=1, gust=1.0),
        # propagation alone: depth refraction on a regional grid
        _case("propags", 600, 450, name="regional_propags", dlat=0.2, dlon=0.2),
        # propagation with tidal currents: frequency shift and refraction by both
        _case("propags", 300, 225, name="currents_propags", dlat=0.2, dlon=0.2, refr_c=True, pad=1),
        # the flagship: one source step of the 0.1 degree regional forecast
        _case("step", 1200, 900, name="regional_step_st6", dlat=0.1, dlon=0.1),
        # a global forecast, ST4, sub-stepped near the poles
        _case("step", 720, 340, name="global_step_st4", lat0=-85.0, lon0=0.0, dlat=0.5, dlon=0.5, land=0.35, ml=35,
              iphys=1, idelt=900, idelpro=300, dmax=6000.0),
        # an ensemble of uneven members advanced together from one captured graph
        _case("ensemble", 260, 200, name="ensemble_step", members=8,
              **dict(deep, lat0=-40.0, lon0=-150.0, dlat=0.4, dlon=0.4)),
        # one iteration of a variational assimilation of Hs: forward and adjoint
        _case("window", 200, 150, name="assimilation_window_st4", dlat=0.6, dlon=0.6, iphys=1, passes=2),
        # an output time step: all integrated parameters and the wind sea / swell split
        _case("output", 400, 300, name="integrated_output", pad=5),
        # the drop-in step of a program that keeps its spectrum in host memory
        _case("hosted", 240, 180, name="hosted_step_st6", dlat=0.5, dlon=0.5),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "implsch", "implsch", "implsch", "propags", "propags", "ensemble", "window",
                       "output", "hosted"])
    most = dict(step=400000, implsch=190000, propags=190000, ensemble=50000, window=21000, output=84000,
                hosted=30000)[kind]
    n = _logint(rng, 2000 if kind == "ensemble" else 100, most)
    nx = max(8, int(math.sqrt(n / 0.7 * rng.uniform(0.8, 1.8))))
    ny = max(6, min(400, int(n / 0.7 / nx)))
    res = min(rng.choice([0.1, 0.25, 0.5, 1.0]), 100.0 / ny, 350.0 / nx)
    shallow = rng.random() < 0.7
    kl, ml, fr1 = rng.choice([(24, 25, 0.04177), (36, 30, 0.0345), (36, 35, 0.0345), (30, 29, 0.0345)])
    idelpro = rng.choice([60, 120]) if res < 0.3 else rng.choice([120, 300])
    c = _case(kind, nx, ny, lat0=-0.5 * ny * res + rng.uniform(-8, 8), lon0=rng.uniform(-180, 0), dlat=res, dlon=res,
              land=rng.choice([0.05, 0.1, 0.3, 0.4]), kl=kl, ml=ml, fr1=fr1, iphys=rng.choice([1, 2]), shallow=shallow,
              refr_d=shallow and rng.random() < 0.8, idelt=600, idelpro=idelpro, dmin=10.0 if shallow else 4000.0,
              dmax=5000.0 if shallow else 4000.0, gust=rng.choice([0.0, 0.0, 1.5]), pad=rng.choice([0, 0, 1, 3, 17]))
    if kind == "propags":
        c["refr_c"] = rng.random() < 0.3
        c["refr_d"] = c["refr_d"] or (c["refr_c"] and shallow)
    if kind == "implsch":
        c["f64"] = nx * ny < 4000 and rng.random() < 0.3
        c["isnonlin"] = int(shallow and rng.random() < 0.15)
    if kind == "ensemble":
        c["members"] = rng.randint(3, 8)
    if kind == "window":
        c["passes"] = rng.randint(1, 2)
    return c


# ---------------------------------------------------------------- synthetic inputs

def _smooth(gen, nx, ny, sigma):
    """Unit-variance Gaussian random field of correlation length sigma cells."""
    z = torch.randn(nx, ny, generator=gen, dtype=torch.float64)
    kx, ky = torch.fft.fftfreq(nx, dtype=torch.float64), torch.fft.rfftfreq(ny, dtype=torch.float64)
    damp = torch.exp(-2.0 * (math.pi * sigma) ** 2 * (kx[:, None] ** 2 + ky[None, :] ** 2))
    f = torch.fft.irfft2(torch.fft.rfft2(z) * damp, s=(nx, ny))
    f = f - f.mean()
    return (f / (f.std() + 1e-30)).numpy()


def _unit(x):
    return (x - x.min()) / (x.max() - x.min() + 1e-30)


def _grid(c, sea):
    """Neighbour tables and metric of a regular latitude-longitude grid: sea
    points numbered south to north, west to east, from 1; 0 is land."""
    nx, ny = sea.shape
    row = sea.T
    num = np.zeros((ny, nx), np.int32)
    num[row] = np.arange(1, int(row.sum()) + 1)
    k, i = np.nonzero(row)
    around = abs(nx * c["dlon"] - 360.0) < 0.5 * c["dlon"]
    west = np.where(i > 0, num[k, i - 1], num[k, nx - 1] if around else 0)
    east = np.where(i < nx - 1, num[k, (i + 1) % nx], num[k, 0] if around else 0)
    south = np.where(k > 0, num[np.maximum(k - 1, 0), i], 0)
    north = np.where(k < ny - 1, num[np.minimum(k + 1, ny - 1), i], 0)
    lat = np.float32((c["lat0"] + c["dlat"] * np.arange(ny)) * PI / 180.0)
    dellam = np.full(ny, np.float32(c["dlon"] * CIRC / 360.0), np.float32)
    n = len(k)
    return dict(nsea=n, klat=np.stack([south, north, south, north]).astype(np.int32).ravel(),
                klon=np.stack([west, east]).astype(np.int32).ravel(), wlat=np.ones(2 * n, np.float32),
                kfromij=(k + 1).astype(np.int32), sinph=np.sin(lat), cosph=np.cos(lat), dellam=dellam,
                delphi=float(np.float32(c["dlat"] * CIRC / 360.0)))


def _inputs(c, seed):
    """Grid and fields of one model: all float32 numpy arrays over sea points."""
    gen = torch.Generator().manual_seed(int(seed) * 7919 + 13)
    nx, ny = c["nx"], c["ny"]
    cells = max(2.0, min(nx, ny) / 45.0)
    noise = _smooth(gen, nx, ny, cells)
    sea = noise < np.quantile(noise, 1.0 - c["land"])
    g = _grid(c, sea)
    pick = lambda a: np.ascontiguousarray(a.T[sea.T]).astype(np.float32)
    depth = c["dmin"] * (c["dmax"] / c["dmin"]) ** _unit(_smooth(gen, nx, ny, 2.0 * cells))
    speed = 4.0 + 17.0 * _unit(_smooth(gen, nx, ny, cells))
    wdir = ZPI * _unit(_smooth(gen, nx, ny, 1.5 * cells))
    fp = 0.075 + 0.16 * _unit(_smooth(gen, nx, ny, cells))
    sdir = ZPI * _unit(_smooth(gen, nx, ny, 2.0 * cells))
    cur_u, cur_v = 0.4 * _smooth(gen, nx, ny, 2.0 * cells), 0.4 * _smooth(gen, nx, ny, 2.0 * cells)
    w = dict(grid=g, n=g["nsea"], depth=pick(depth), u10=pick(speed), udir=pick(wdir), fp=pick(fp), sdir=pick(sdir),
             cur_u=pick(cur_u) if c["refr_c"] else None, cur_v=pick(cur_v) if c["refr_c"] else None)
    n = w["n"]
    rnd = torch.rand(2, n, generator=gen).numpy()
    w["roairn"] = (1.2 + 0.06 * rnd[0]).astype(np.float32)
    w["wstar"] = (c["gust"] * rnd[1]).astype(np.float32)
    us = (w["u10"] * np.sqrt(1e-3 * (0.8 + 0.08 * w["u10"]))).astype(np.float32)
    w["tauw"] = (0.4 * us * us).astype(np.float32)
    return w


def _spectrum(c, w, device, dtype):
    """Sea state (ML, KL, N): a JONSWAP wind sea with cos^2 spreading about the
    wind and a swell of another direction."""
    t = lambda a: torch.tensor(a, device=device, dtype=torch.float32)
    fr = torch.tensor(c["fr1"] * 1.1 ** np.arange(c["ml"]), device=device, dtype=torch.float32)[:, None]
    th = torch.tensor((np.arange(c["kl"]) + 0.5) * 2 * math.pi / c["kl"], device=device, dtype=torch.float32)[:, None]

    def one(fp, alpha, gamma, direction, power):
        x = (1.25 * (fp / fr) ** 4).clamp(max=50.0)
        e = alpha * G ** 2 / ZPI ** 4 * fr ** -5 * torch.exp(-x)
        a = (0.5 * ((fr / fp - 1.0) / torch.where(fr > fp, 0.09, 0.07)) ** 2).clamp(max=99.0)
        e = e * torch.exp(math.log(gamma) * torch.exp(-a))
        return e, (2.0 / math.pi) * torch.cos(th - direction).clamp(min=0.0) ** power

    e1, d1 = one(t(w["fp"])[None], 0.012, 3.3, t(w["udir"])[None], 2)
    e2, d2 = one(0.6 * t(w["fp"])[None], 0.0008, 4.0, t(w["sdir"])[None], 6)
    return (e1[:, None] * d1[None] + e2[:, None] * d2[None]).to(dtype)


def _config(c, delphi):
    return make_config(c["kl"], c["ml"], c["fr1"], c["iphys"], c["idelt"], c["idelpro"], delphi,
                       shallow_run=c["shallow"], spherical_run=True, refraction_d_run=c["refr_d"],
                       refraction_c_run=c["refr_c"], isnonlin=c["isnonlin"],
                       betamax=1.42 if c["iphys"] == 1 else 1.20, precision=8 if c["f64"] else 4)


def _member(c, k):
    """Member k of an ensemble: its own size, spectral grid and physics."""
    f = (1.0, 0.35, 0.6, 0.22, 0.8, 0.3, 0.5, 0.15)[k % 8]
    m = dict(c, nx=max(8, int(c["nx"] * f)), ny=max(6, int(c["ny"] * f)), iphys=1 + k % 2)
    if k % 3 == 1:
        m.update(kl=36, ml=30, fr1=0.0345)
    return m


# ---------------------------------------------------------------- prepare and run

def _stream():
    h = torch.cuda.current_stream().cuda_stream
    return h if h else 1  # the library's name for the legacy default stream


def _model(c, w):
    m = WamModel(_config(c, w["grid"]["delphi"]))
    m.set_grid(w["grid"])
    m.set_depth(w["depth"])
    if c["refr_c"]:
        m.set_current(w["cur_u"], w["cur_v"])
    m.prepare_propagation()
    m.prepare_source()
    return m


def _fields(c, w):
    dt = torch.float64 if c["f64"] else torch.float32
    ld = w["n"] + c["pad"]
    f = torch.zeros((c["ml"], c["kl"], ld), device=DEV, dtype=dt)
    f[:, :, :w["n"]] = _spectrum(c, w, DEV, dt)
    t = lambda a: torch.tensor(a, device=DEV, dtype=dt)
    return dict(f=f, u10=t(w["u10"]), udir=t(w["udir"]), tauw=t(w["tauw"]), ustar=torch.zeros(w["n"], device=DEV, dtype=dt),
                z0=torch.zeros(w["n"], device=DEV, dtype=dt), roairn=t(w["roairn"]), wstar=t(w["wstar"]))


def _observations(c, w, seed):
    rng = np.random.default_rng(seed + 77)
    pts = np.sort(rng.choice(w["n"], max(1, w["n"] // 40), replace=False))
    return pts, (0.5 + 3.0 * rng.random((max(1, c["passes"]), len(pts)))).astype(np.float32)


def prepare(case, seed):
    c = case
    s = dict(case=c, nprop=c["idelt"] // c["idelpro"])
    if c["kind"] == "ensemble":
        s["models"], s["state"] = [], []
        for k in range(c["members"]):
            mc = _member(c, k)
            w = _inputs(mc, seed + 1000 * k)
            s["models"].append(_model(mc, w))
            s["state"].append(_fields(mc, w))
        s["batch"] = WamBatch(s["models"])
        for k, d in enumerate(s["state"]):
            s["batch"].set_member(k, d["f"], torch.empty_like(d["f"]), *[d[q] for q in ("u10", "udir", "tauw", "ustar",
                                                                                      "z0", "roairn", "wstar")])
        torch.cuda.synchronize()
        s["batch"].capture(stream=None)
        s["batch"].sync()
        return s
    w = _inputs(c, seed)
    s["model"] = _model(c, w)
    if c["kind"] == "hosted":
        pin = lambda a: torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()
        f = torch.empty((c["ml"], c["kl"], w["n"]), pin_memory=True)
        f.copy_(_spectrum(c, w, DEV, torch.float32))
        s.update(f=f.numpy(), pinned=f, n=w["n"], ustar=pin(np.zeros(w["n"], np.float32)),
                 z0=pin(np.zeros(w["n"], np.float32)),
                 **{q: pin(w[q]) for q in ("u10", "udir", "tauw", "roairn", "wstar")})
        return s
    s.update(_fields(c, w))
    if c["kind"] in ("step", "propags", "window"):
        s["scratch"] = torch.empty_like(s["f"])
    if c["kind"] == "output":
        s["block"] = torch.zeros((40, w["n"]), device=DEV)
        us = w["u10"] * np.sqrt(1e-3 * (0.8 + 0.08 * w["u10"]))
        s["ustar"].copy_(torch.tensor(us))
        s["z0"].copy_(s["ustar"] ** 2 * (0.012 / G))
    if c["kind"] == "window":
        pts, obs = _observations(c, w, seed)
        s["points"], s["obs"] = torch.tensor(pts, device=DEV), torch.tensor(obs, device=DEV)
        s["dfim"] = torch.tensor(s["model"].table("DFIM"), device=DEV)
        s["model"].checkpoint_reserve(c["passes"], s["f"].shape[-1])
        s["work"], s["work_tauw"] = torch.empty_like(s["f"]), torch.empty_like(s["tauw"])
        s["lam"] = torch.empty_like(s["f"])
    return s


def _hs(f, dfim, points):
    return 4.0 * torch.sqrt((f[:, :, points].sum(dim=1) * dfim[:, None]).sum(dim=0))


def run(s):
    c, q = s["case"], _stream() if s["case"]["kind"] not in ("hosted", "ensemble") else None
    if c["kind"] == "step":
        s["model"].step_dev(s["f"], s["nprop"], s["u10"], s["udir"], s["tauw"], s["ustar"], s["z0"], s["roairn"],
                            s["wstar"], scratch=s["scratch"], stream=q)
        return dict(f=s["f"], tauw=s["tauw"], ustar=s["ustar"], z0=s["z0"])
    if c["kind"] == "implsch":
        s["model"].implsch_dev(s["f"], s["u10"], s["udir"], s["tauw"], s["ustar"], s["z0"], s["roairn"], s["wstar"],
                               stream=q)
        return dict(f=s["f"], tauw=s["tauw"], ustar=s["ustar"], z0=s["z0"])
    if c["kind"] == "propags":
        s["model"].propags_dev(s["f"], scratch=s["scratch"], stream=q)
        return dict(f=s["f"])
    if c["kind"] == "ensemble":
        s["batch"].step(stream=_stream())
        return [dict(f=d["f"], tauw=d["tauw"], ustar=d["ustar"]) for d in s["state"]]
    if c["kind"] == "output":
        m = s["model"]
        m.output_parameters_dev(s["f"], s["u10"], s["udir"], s["tauw"], s["ustar"], s["z0"], block=s["block"], stream=q)
        m.output_swell_dev(s["f"], s["udir"], s["ustar"], s["block"], stream=q)
        return dict(block=s["block"])
    if c["kind"] == "hosted":
        s["model"].step(s["f"], s["nprop"], s["u10"], s["udir"], s["tauw"], s["ustar"], s["z0"], s["roairn"], s["wstar"])
        return dict(f=s["f"], tauw=s["tauw"], ustar=s["ustar"], z0=s["z0"])
    # window: forward from the background with checkpoints, then the adjoint
    m, f, lam, pts, dfim = s["model"], s["work"], s["lam"], s["points"], s["dfim"]
    f.copy_(s["f"])
    s["work_tauw"].copy_(s["tauw"])
    grads = []
    for p in range(c["passes"]):
        m.step_ckpt_dev(p, f, s["nprop"], s["u10"], s["udir"], s["work_tauw"], s["ustar"], s["z0"], s["roairn"],
                        s["wstar"], scratch=s["scratch"], stream=q)
        hs = _hs(f, dfim, pts)
        # dJ/dF(m, k, point) of (Hs - Hs_obs)^2
        grads.append((16.0 * (hs - s["obs"][p]) / hs)[None, :] * dfim[:, None])
    lam.zero_()
    lam_t, lam_u = torch.zeros_like(s["tauw"]), [torch.empty_like(s["u10"]) for _ in grads]
    for p in reversed(range(c["passes"])):
        lam[:, :, pts] += grads[p][:, None, :]
        m.step_adj_dev(p, s["nprop"], lam, lam_t, lam_u[p], s["udir"], s["roairn"], s["wstar"], scratch=s["scratch"],
                       stream=q)
    return dict(grad_f=lam, grad_tauw=lam_t, grad_u10=lam_u)


# ---------------------------------------------------------------- work

def _sea(c):
    n = c["nx"] * c["ny"]
    return n - int(round(c["land"] * n))


def _flops(c, n, props, sources):
    """Floating-point operations: 34 per bin of a propagation sub-step, 260
    (ST6) or 560 (ST4) per bin of the source terms, an add, a product or a
    function call each one."""
    return float(n) * c["kl"] * c["ml"] * (34.0 * props + (260.0 if c["iphys"] == 2 else 560.0) * sources)


def work(case):
    c = case
    if c["kind"] == "ensemble":
        parts = [_member(c, k) for k in range(c["members"])]
        w = [work(dict(p, kind="step", members=0)) for p in parts]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    n, size = _sea(c), 8 if c["f64"] else 4
    spec = float(n) * c["kl"] * c["ml"] * size
    fields = float(n) * size
    nprop = c["idelt"] // c["idelpro"]
    if c["kind"] == "propags":
        return {"bytes": 2 * spec + 12 * fields, "flops": _flops(c, n, 1, 0)}
    if c["kind"] == "implsch":
        return {"bytes": 2 * spec + 12 * fields, "flops": _flops(c, n, 0, 1)}
    if c["kind"] == "output":
        return {"bytes": spec + 38 * fields, "flops": float(n) * c["kl"] * c["ml"] * 12.0}
    if c["kind"] == "window":
        # forward and adjoint each once per pass, the adjoint at twice the forward's operations
        return {"bytes": c["passes"] * 2 * (2 * spec * (nprop + 1) + 12 * fields),
                "flops": 3.0 * c["passes"] * _flops(c, n, nprop, 1)}
    return {"bytes": 2 * spec * (nprop + 1) + 12 * fields, "flops": _flops(c, n, nprop, 1)}


# ---------------------------------------------------------------- float64 restatement

def _t64(a):
    return torch.tensor(np.asarray(a, np.float64), device=DEV, dtype=torch.float64)


@functools.lru_cache(maxsize=8)
def _swell_friction(kappa=0.40):
    """Friction factor of the oscillatory boundary layer over log10(a/z0):
    fixed point of f = 0.08 / (ker^2 + kei^2), the Kelvin functions from
    K0(z) = int_0^inf exp(-z cosh t) dt (trapezoidal rule)."""
    lo, step = 0.3, (8.0 - 0.3) / 200
    abr = np.exp((lo + np.arange(1, 201) * step) * math.log(10.0))
    fact = 1.0 / abr / (21.2 * kappa)
    f, dz = np.full(200, 0.05), np.zeros(200)
    h = 0.02
    t = np.arange(0, 900) * h
    wt = np.full(900, h)
    wt[0] = h / 2
    for _ in range(100):
        f0, dz0 = f, dz
        dz = fact * f ** -0.5
        zr = 2.0 * np.sqrt(dz) * 0.5 * math.sqrt(2.0)
        ch = np.minimum(np.cosh(t), 1e6)
        k0 = (np.exp(-np.minimum((zr[:, None]) * ch[None], 700.0)) * np.exp(-1j * (zr[:, None] * ch[None]))) @ wt
        f = 0.5 * (f0 + 0.08 / np.abs(k0) ** 2)
        dz = 0.5 * (dz0 + dz)
    return f


def _tables(c, delphi):
    """The static tables in float64 (frequency grid, depth tables, minimum
    energy, DIA, saturation weights, 10 Hz axis)."""
    kl, ml = c["kl"], c["ml"]
    T = dict(kl=kl, ml=ml)
    fr = np.empty(ml)
    fr[0] = c["fr1"]
    for m in range(1, ml):
        fr[m] = 1.1 * fr[m - 1]
    delth = ZPI / kl
    th = (np.arange(kl) + 0.5) * delth
    df = np.empty(ml)
    df[0], df[-1] = 0.05 * fr[0], 0.05 * fr[ml - 2]
    df[1:-1] = 0.05 * (fr[1:-1] + fr[:-2])
    T.update(fr=fr, df=df, delth=delth, th=th, dfim=df * delth, dfimofr=df * delth / fr)
    tail = (-(delth / -4.0 * fr[-1]), delth / 5.0, -(delth / -3.0 * fr[-1] ** 2), -(delth / -2.0 * fr[-1] ** 3))
    T["mo_tail"], T["mm1_tail"], T["mp1_tail"], T["mp2_tail"] = tail
    rho = 1000.0 * G * delth * math.log(1.1) * fr
    rho[0] *= 0.5
    rho[-1] *= 0.5
    T["rhowg"] = rho
    tfak, tcg, tsi = (np.zeros((ml, NDEPTH)) for _ in range(3))
    for m in range(ml):
        om = ZPI * fr[m]
        for j in range(NDEPTH):
            d = DEPTHA * DEPTHD ** j
            ak, prev = max(om * om / (4 * G), om / (2 * math.sqrt(G * d))), 1e4
            while abs(prev - ak) > 1e-4 * ak:
                bo = d * ak
                if bo > 40.0:
                    ak = om * om / G
                    break
                prev = ak
                t = G * ak * math.tanh(bo)
                st = math.sqrt(t)
                ak = ak + (om - st) * st * 2.0 / (t / ak + G * bo / math.cosh(bo) ** 2)
            tfak[m, j] = ak
            x = ak * d
            if x <= 10.0:
                tcg[m, j] = 0.5 * math.sqrt(G * math.tanh(x) / ak) * (1 + 2 * x / math.sinh(2 * x))
                tsi[m, j] = om / math.sinh(2 * x)
            else:
                tcg[m, j] = G / (4 * PI) / fr[m]
    T.update(tfak=tfak, tcg=tcg, tsi=tsi)
    # minimum energy per wind speed class of 0.25 m/s
    fetch = min(0.5 * delphi, 25000.0)
    u = 0.25 * np.arange(1, 301)
    f = np.maximum(0.13, 2.84 * (G * fetch / u ** 2) ** -0.3)
    f = np.minimum(f, fr[-1] / (G / u))
    alph, fpk = 0.01 * np.maximum(0.0081, 0.033 * f ** (2.0 / 3.0)), f * G / u
    arg = 1.25 * (fpk[None] / fr[:, None]) ** 4
    e = np.where(arg < 50, alph * G ** 2 / ZPI ** 4 * fr[:, None] ** -5 * np.exp(-np.minimum(arg, 50)), 0.0)
    a2 = np.where(fr[:, None] > fpk, 0.5 / 0.09 ** 2, 0.5 / 0.07 ** 2) * (fr[:, None] / fpk - 1) ** 2
    e = np.where((arg < 50) & (a2 < 99), e * np.exp(math.log(3.0) * np.exp(-np.minimum(a2, 99))), e)
    T["flmin"] = np.maximum(e, 1e-6)
    # DIA geometry: lambda = 0.25 on a grid of ratio 1.1
    lam = 0.25
    c3 = (1 + 2 * lam + 2 * lam ** 3) / (1 + lam) ** 2
    d1 = -180.0 / PI * math.acos(c3)
    xf = ((1 + lam) / (1 - lam)) ** 4
    d2 = 180.0 / PI * math.acos(math.sqrt(1 - xf + xf * c3 * c3))
    cl1, cl2 = d1 / (delth * 180.0 / PI), d2 / (delth * 180.0 / PI)
    T["rot1"], T["rot2"] = int(cl1), int(cl2)
    T["s1"], T["s2"] = (-1 if cl1 < 0 else 1), (-1 if cl2 < 0 else 1)
    T["acl1"], T["acl2"] = abs(cl1 - int(cl1)), abs(cl2 - int(cl2))
    T["dal1"], T["dal2"] = 1 / (1 + lam) ** 4, 1 / (1 - lam) ** 4
    T["co"] = 1.1
    # saturation window (80 degrees either side)
    half = min(int(math.floor(80 * PI / 180.0 / delth + 0.5)), kl // 2 - 1)
    trunc = min(max(th[0] + 80 * PI / 180.0 - (th[half] - 0.5 * delth), 0.0), delth)
    off = np.arange(-half, half + 1)
    T["sat"] = [(int(o), (trunc if abs(o) == half else delth) * math.cos(o * delth) ** 2) for o in off]
    nk10 = max(ml, int(math.ceil(math.log(10.0 / fr[0]) / math.log(1.1))) + 1)
    sig10 = ZPI * fr[0] * 1.1 ** np.arange(nk10)
    ds10 = 0.5 * sig10 * (1.1 - 1 / 1.1)
    ds10[0], ds10[-1] = 0.5 * sig10[0] * 0.1, 0.5 * sig10[-1] * 0.1 / 1.1
    T.update(nk10=nk10, sig10=sig10, ds10=ds10)
    return T


def _depth_class(d):
    return np.clip(np.floor(np.log(d / DEPTHA) / math.log(DEPTHD) + 1.5), 1, NDEPTH).astype(np.int64)


class _Exact64:
    """PROPAGS, IMPLSCH and the integrated output of one model in float64."""

    def __init__(self, c, w):
        self.c, self.w, self.g = c, w, w["grid"]
        self.T = T = _tables(c, self.g["delphi"])
        n = w["n"]
        cfg = _config(c, self.g["delphi"])
        self.cfg = {k: cfg[k] for k in ("betamax", "zalp", "alpha", "tauwshelter", "cdfac")}
        depth = w["depth"].astype(np.float64)
        self.ind = _depth_class(depth) if c["shallow"] else np.ones(n, np.int64)
        self.tfak, self.tcg = _t64(T["tfak"]), _t64(T["tcg"])
        self.iind = torch.tensor(self.ind - 1, device=DEV)

    # ---- propagation ------------------------------------------------------
    def _coefficients(self):
        c, g, T, w = self.c, self.g, self.T, self.w
        n = w["n"]
        idx = lambda a: torch.tensor(a, device=DEV, dtype=torch.int64)
        S, N = idx(g["klat"][:n]), idx(g["klat"][n:2 * n])
        W, E = idx(g["klon"][:n]), idx(g["klon"][n:])
        row = g["kfromij"] - 1
        dco_row = 1.0 / g["cosph"].astype(np.float64)
        dco = _t64(dco_row[row])
        dcol = torch.cat([torch.ones(1, device=DEV, dtype=torch.float64), dco])
        ps = torch.where(S > 0, dco / dcol[S], torch.ones_like(dco))
        pn = torch.where(N > 0, dco / dcol[N], torch.ones_like(dco))
        delphi, dellam = g["delphi"], float(g["dellam"][0])
        dt = float(c["idelpro"])
        delph0, delth0 = 0.5 * dt / delphi, 0.5 * dt / (T["delth"] * RAD_E)
        delthr = 0.5 * dt / T["delth"]
        d0 = dt * dco / dellam * (0.5 if (c["shallow"] or c["refr_c"]) else 1.0)
        if not c["shallow"] and c["refr_c"]:
            d0 = 0.5 * dt * dco / dellam
        dr = _t64(g["sinph"].astype(np.float64)[row]) * dco
        self.nb = (S, N, W, E)
        land = torch.zeros(1, device=DEV, dtype=torch.float64)
        pad = lambda a, v=0.0: torch.cat([land + v, a])

        def gradient(a):
            lat = torch.where((S > 0) & (N > 0), (a[N] - a[S]) / (2 * delphi), 0.0)
            lon = torch.where((W > 0) & (E > 0), (a[E] - a[W]) / (2 * dellam), 0.0)
            return lat, lon * dco

        D = pad(_t64(w["depth"]), 999.0)
        ddphi, ddlam = gradient(D)
        mean, cnt = 4 * D[1:], torch.full((n,), 4.0, device=DEV, dtype=torch.float64)
        both = (S > 0) & (N > 0)
        mean, cnt = mean + torch.where(both, D[S] + D[N], 0.0), cnt + 2.0 * both
        both = (W > 0) & (E > 0)
        mean, cnt = mean + torch.where(both, D[W] + D[E], 0.0), cnt + 2.0 * both
        indg = torch.tensor(_depth_class((mean / cnt).cpu().numpy()) - 1, device=DEV)
        ind = torch.cat([torch.full((1,), NDEPTH - 1, device=DEV, dtype=torch.int64), self.iind])
        sn, cs = _t64(np.sin(T["th"]))[:, None], _t64(np.cos(T["th"]))[:, None]
        sp, sm = delth0 * (sn + sn.roll(-1, 0)), delth0 * (sn + sn.roll(1, 0))
        isn, ics = sn >= 0, cs >= 0
        if c["refr_c"]:
            U, V = pad(_t64(w["cur_u"])), pad(_t64(w["cur_v"]))
            duphi, dulam = gradient(U)
            dvphi, dvlam = gradient(V)
        ml = T["ml"]
        tsi = _t64(T["tsi"])
        z = torch.zeros((), device=DEV, dtype=torch.float64)
        for m in range(ml):
            o = {}
            gom = G / (4 * PI * T["fr"][m])
            cg = self.tcg[m][ind] if c["shallow"] else torch.full((n + 1,), gom, device=DEV, dtype=torch.float64)
            c0, cS, cN, cW, cE = cg[1:], cg[S], cg[N], cg[W], cg[E]
            ts = tsi[m][indg] if c["shallow"] else None
            if not c["refr_c"]:
                sda, cda = sn.abs(), (cs * delph0).abs()
                if c["shallow"]:
                    k1, k2 = c0 + ps * cS, c0 + pn * cN
                    o["lat"] = cda * torch.where(ics, k1, k2)
                    o["lon"] = sda * (torch.where(isn, cW, cE) + c0) * d0
                    tc = 1 - cda * torch.where(ics, k2, k1) - sda * (torch.where(isn, cE, cW) + c0) * d0
                    dtp, dtm = dr * c0 * sp, dr * c0 * sm
                    if c["refr_d"]:
                        thdd = (sn * ddphi - cs * ddlam) * ts
                        dtp = dtp + (thdd + thdd.roll(-1, 0)) * delthr
                        dtm = dtm + (thdd + thdd.roll(1, 0)) * delthr
                    tc = tc - torch.maximum(z, dtp) + torch.minimum(z, dtm)
                    o["th1"], o["th2"], o["sum"] = -torch.minimum(z, dtp), torch.maximum(z, dtm), tc
                else:
                    dle = sda * d0
                    o["lat"] = gom * cda * (torch.where(ics, ps, pn) + 1)
                    o["lon"] = gom * dle
                    dtp, dtm = dr * sp, dr * sm
                    tc = cda * (torch.where(ics, pn, ps) + 1) + dle + torch.maximum(z, dtp) - torch.minimum(z, dtm)
                    o["th1"], o["th2"] = -(gom * torch.minimum(z, dtp)), gom * torch.maximum(z, dtm)
                    o["sum"] = 1 - gom * tc
            else:
                u0, uW, uE, v0, vS, vN = U[1:], U[W], U[E], V[1:], V[S], V[N]
                w1, w2 = u0 + sn * c0, (v0 + cs * c0) * delph0
                dlw, dle = (w1 + uW + sn * cW) * d0, (w1 + uE + sn * cE) * d0
                dps, dpn = w2 + ps * (vS + cs * cS) * delph0, w2 + pn * (vN + cs * cN) * delph0
                tc = 1 - torch.maximum(z, dle) + torch.minimum(z, dlw) - torch.maximum(z, dpn) + torch.minimum(z, dps)
                o["lonW"], o["lonE"] = torch.maximum(z, dlw), -torch.minimum(z, dle)
                o["latS"], o["latN"] = torch.maximum(z, dps), -torch.minimum(z, dpn)
                thdd = sn * sn * duphi + sn * cs * dvphi - sn * cs * dulam - cs * cs * dvlam
                if c["shallow"]:
                    thdd = thdd + (sn * ddphi - cs * ddlam) * ts
                dtp = sp * dr * c0 + (thdd + thdd.roll(-1, 0)) * delthr
                dtm = sm * dr * c0 + (thdd + thdd.roll(1, 0)) * delthr
                tc = tc - torch.maximum(z, dtp) + torch.minimum(z, dtm)
                o["th1"], o["th2"] = -torch.minimum(z, dtp), torch.maximum(z, dtm)
                b = -(sn * cs * duphi) - cs * cs * dvphi - sn * sn * dulam - sn * cs * dvlam
                if c["shallow"]:
                    mp, mm = min(m + 1, ml - 1), max(m - 1, 0)
                    drift = v0 * ddphi + u0 * ddlam
                    at = lambda q: (b * self.tcg[q][self.iind] + drift * tsi[q][indg]) * self.tfak[q][indg]
                    f0 = 0.5 * dt / (0.1 * ZPI)
                    dop, dom = (at(m) + at(mp)) * f0 / T["fr"][m], (at(m) + at(mm)) * f0 / T["fr"][mm]
                    o["sg1"], o["sg2"] = -torch.minimum(z, dop) / 1.1, torch.maximum(z, dom) * 1.1
                    tc = tc - torch.maximum(z, dop) + torch.minimum(z, dom)
                else:
                    dom = b * (0.5 * dt * 2.1 / 0.2)
                    o["sg1"], o["sg2"] = -torch.minimum(z, dom) / 1.1, torch.maximum(z, dom) * 1.1
                    tc = tc - dom.abs()
                o["sum"] = tc
            yield o

    def counter(self):
        most = 0.0
        for o in self._coefficients():
            most = max([most, float(1 - o["sum"].min())] + [float(v.max()) for k, v in o.items() if k != "sum"])
        return int(math.ceil(most)) if most > 0.999 else 1

    def propagate(self, f, cnt):
        """One propagation time step of cnt sub-steps; f (ML, KL, N) float64."""
        for _ in range(cnt):
            new = torch.empty_like(f)
            ml, kl, n = f.shape
            for m, o in enumerate(self._coefficients()):
                if cnt != 1:
                    o = {k: (1 - (1 - v) / cnt if k == "sum" else v / cnt) for k, v in o.items()}
                F = torch.cat([torch.zeros((kl, 1), device=DEV, dtype=f.dtype), f[m]], 1)
                S, N, W, E = self.nb
                ics, isn = _t64(np.cos(self.T["th"]))[:, None] >= 0, _t64(np.sin(self.T["th"]))[:, None] >= 0
                v = o["sum"] * f[m] + o["th1"] * f[m].roll(-1, 0) + o["th2"] * f[m].roll(1, 0)
                if "lat" in o:
                    v = v + o["lat"] * torch.where(ics, F[:, S], F[:, N]) + o["lon"] * torch.where(isn, F[:, W], F[:, E])
                else:
                    v = v + o["latS"] * F[:, S] + o["latN"] * F[:, N] + o["lonW"] * F[:, W] + o["lonE"] * F[:, E]
                    v = v + o["sg1"] * f[min(m + 1, ml - 1)] + o["sg2"] * f[max(m - 1, 0)]
                new[m] = v
            f = new
        return f

    # ---- source terms -----------------------------------------------------
    def implsch(self, f, tauw):
        """One source step; returns (f, tauw, ustar, z0)."""
        n = self.w["n"]
        step = max(1, int(1.5e8 // (f.shape[0] * f.shape[1])))
        out = [self._implsch(f[:, :, i:i + step], tauw[i:i + step], slice(i, min(n, i + step)))
               for i in range(0, n, step)]
        return tuple(torch.cat([o[q] for o in out], -1) for q in range(4))

    def _implsch(self, F, tauw, sl):
        c, T, w, cf = self.c, self.T, self.w, self.cfg
        ml, kl = T["ml"], T["kl"]
        u10, udir, roairn, wstar, depth = (_t64(w[q][sl]) for q in ("u10", "udir", "roairn", "wstar", "depth"))
        ind = self.iind[sl]
        fr, dfim, dfimofr = _t64(T["fr"])[:, None], _t64(T["dfim"])[:, None], _t64(T["dfimofr"])[:, None]
        th = _t64(T["th"])[:, None]
        sh = c["shallow"]
        tfak, tcg = self.tfak[:, ind], self.tcg[:, ind]
        sig = ZPI * fr
        ju = torch.floor(u10 / 0.25 + 0.5).clamp(1, 300).long() - 1
        self.x = dict(u10=u10, udir=udir, roairn=roairn, wstar=wstar, tfak=tfak, tcg=tcg, sig=sig, fr=fr, th=th)

        def integrals(F, mask, akm):
            t, tw = F.sum(1), torch.where(mask, F, 0.0).sum(1)
            e = (t * dfim).sum(0) + T["mo_tail"] * t[-1]
            fm = (t * dfimofr).sum(0) + T["mm1_tail"] * t[-1]
            ew = (tw * dfim).sum(0) + T["mo_tail"] * tw[-1]
            fw = (tw * dfimofr).sum(0) + T["mm1_tail"] * tw[-1]
            e, ew = e.clamp(min=1e-12), ew.clamp(min=1e-12)
            ak = None
            if akm:
                del2 = math.sqrt(G) / ZPI
                wm = (t / tfak.sqrt() * dfim).sum(0) + T["mm1_tail"] * del2 * t[-1]
                ak = torch.where(e > 1e-12, (e / wm) ** 2, 1.0)
            return e, e / fm.clamp(min=1e-12), ak, ew / fw.clamp(min=1e-12)

        def cut(fm, fmws, ustar):
            if c["iphys"] == 2:
                f1 = 1.0 / math.log(1.1)
                f2 = 1.0 - math.log(ZPI * T["fr"][0]) * f1
                hi = torch.maximum(6 * ZPI * fm, 4 * G / 28 / ustar)
                nkh1 = ((f2 + f1 * torch.log(hi.clamp(min=1e-7))).trunc().clamp(max=ml) + 1).clamp(max=ml)
                hi = hi.clamp(max=ZPI * T["fr"][-1])
                m = torch.minimum(nkh1, (f2 + f1 * torch.log(hi.clamp(min=1e-7))).trunc()).clamp(min=2)
                return m.long()
            x = torch.maximum(torch.maximum(fmws, fm) * (2.5 / T["fr"][0]),
                              3 * G / (28 * ZPI * T["fr"][0]) / ustar.clamp(min=1e-6))
            return (torch.floor(torch.log10(x) / math.log10(1.1) + 0.5) + 1).clamp(1, ml).long()

        def tail(F, mij):
            t = 1.0 / tfak ** 3 / tcg if sh else (1.0 / fr ** 5).expand(ml, F.shape[2])
            ref = torch.gather(F, 0, (mij - 1)[None, None, :].expand(1, kl, -1))
            base = torch.gather(t, 0, (mij - 1)[None, :])
            up = torch.arange(ml, device=DEV)[:, None] >= mij[None]
            return torch.where(up[:, None, :], (t / base)[:, None, :] * ref, F)

        akm = sh and c["isnonlin"] == 0
        if c["iphys"] == 1:
            ustar, z0 = self._airsea(tauw)
            _, _, ll, st = self._sinput_ard(F, ustar, z0)
            e, fm, ak, fmws = integrals(F, ll, akm)
            mij = cut(fm, fmws, ustar)
            tauw = self._stresso(F, st, mij, ustar, z0)
            ustar, z0 = self._airsea(tauw)
            F = tail(F, mij)
            S, D, ll, st = self._sinput_ard(F, ustar, z0)
            tauw = self._stresso(F, st, mij, ustar, z0)
            S, D = self._sdissip_ard(F, S, D)
        else:
            ustar, z0 = self._w3flx4()
            S, D, ll, tauw = self._sinput_st6(F, ustar, depth)
            e, fm, ak, fmws = integrals(F, ll, akm)
            mij = cut(fm, fmws, ustar)
            F = tail(F, mij)
            S, D = self._sdissip_st6(F, S, D)
        S, D = self._snonlin(F, S, D, ak, depth)
        if sh:
            sbo = -2.0 * 0.038 / G * tfak / torch.sinh((2 * depth * tfak).clamp(max=50.0))
            S, D = S + sbo[:, None] * F, D + sbo[:, None]
        dt = float(c["idelt"])
        delfl = 5e-7 * G / fr ** 4 * dt
        lim = (ustar * delfl * torch.maximum(fmws, fm))[:, None]
        inc = dt * S / (1 - dt * D).clamp(min=1.0)
        F = F + inc.sign() * torch.minimum(inc.abs(), lim)
        spread = torch.cos(th - udir).clamp(min=0.0) ** 2
        F = torch.maximum(F, _t64(T["flmin"])[:, ju][:, None] * spread[None])
        e, fm, _, fmws = integrals(F, ll, False)
        return tail(F, cut(fm, fmws, ustar)), tauw, ustar, z0

    def _airsea(self, tauw):
        u10, eps = self.x["u10"], 1e-5
        xk, alphaog = 0.40 * u10, self.cfg["alpha"] / G
        old = torch.maximum((u10 * torch.sqrt(8e-4 + 8e-5 * u10)) ** 2, tauw + eps)
        us = old.sqrt()
        um1 = 1 / us.clamp(min=1e-6)
        z0ch = torch.zeros_like(us)
        live = torch.ones_like(us, dtype=torch.bool)
        for _ in range(15):
            x = tauw / old
            zc = alphaog * old / torch.sqrt((1 - x).clamp(min=eps))
            zv = 0.11 * 1.5e-5 * um1
            zt = zc + zv
            xl = 1 / (math.log(10.0) - torch.log(zt))
            zz = um1 * (zc * (2 - 3 * x) / (1 - x) - zv) / zt
            new = us - (us - xk * xl) / (1 - xk * xl ** 2 * zz)
            tn = torch.maximum(new * new, tauw + eps)
            z0ch = torch.where(live, zc, z0ch)
            us = torch.where(live, tn.sqrt(), us)
            done = live & (tn == old)
            old = torch.where(live, tn, old)
            live = live & ~done
            um1 = torch.where(live, 1 / us.clamp(min=1e-6), um1)
        return us, z0ch

    def _w3flx4(self):
        u = self.x["u10"]
        cd = self.cfg["cdfac"] * ((8.058 + 0.967 * u) - 0.016 * u * u) * 1e-4
        us = torch.where(u >= 50.33, 2.026 * math.sqrt(self.cfg["cdfac"]), u * cd.clamp(min=0).sqrt())
        cd = torch.where(u >= 50.33, (us / u) ** 2, cd)
        return us, 10.0 * torch.exp(-0.4 / cd.sqrt())

    def _wsigstar(self, us, z0):
        u = (us / 0.40 * (math.log(10.0) - torch.log(z0))).clamp(min=1.0)
        c1, c2, p1, p2 = 1.03e-3, 0.04e-3, 1.48, -0.21
        c2u, up2 = c2 * u ** p1, u ** p2
        cd, dcd = (c1 + c2u) * up2, (p2 * c1 + (p1 + p2) * c2u) * up2 / u
        return ((1 + 0.5 * u / cd * dcd) / u * (0.5 * 0.40 * self.x["wstar"] ** 3) ** (1.0 / 3.0)).clamp(max=0.1)

    def _sinput_ard(self, F, us, z0):
        x, T, cf, sh = self.x, self.T, self.cfg, self.c["shallow"]
        ml, kl = T["ml"], T["kl"]
        nu, row, kap = 1.5e-5, 1000.0, 0.40
        sn, cs = torch.sin(x["th"]), torch.cos(x["th"])
        t = F.sum(1)
        dfim = _t64(T["dfim"])[:, None]
        tiny = 2.2250738585072014e-308 if self.c["f64"] else 1.1754943508222875e-38
        uorb = 2 * torch.sqrt(tiny + (dfim * x["sig"] ** 2 * t).sum(0))
        aorb = 2 * torch.sqrt(tiny + (dfim * t).sum(0))
        re = 4 / nu * uorb * aorb
        z0noz = torch.maximum(0.11 * 1.5e-5 / us.clamp(min=1e-4), 0.04 * z0.clamp(max=0.0005))
        xi = (torch.log10((aorb / z0noz).clamp(min=3.0)) - 0.3) * (200 / (8.0 - 0.3))
        ind = xi.trunc().clamp(1, 199)
        d1 = (xi - ind).clamp(max=1.0)
        tab = _t64(_swell_friction())
        fww = tab[ind.long() - 1] * (1 - d1) + tab[ind.long()] * d1
        temp2 = fww * uorb
        smooth = 0.5 * torch.tanh((re - 1.5e5) / 3.6e5)
        pturb, pvisc = 0.5 + smooth, 0.5 - smooth
        sg = self._wsigstar(us, z0)
        shelter = abs(cf["tauwshelter"])
        gusts = [(us * (1 + sg)) ** 2, (us * (1 - sg)) ** 2]
        tx, ty = [g * torch.sin(x["udir"]) for g in gusts], [g * torch.cos(x["udir"]) for g in gusts]
        xs, ys = [torch.zeros_like(us) for _ in gusts], [torch.zeros_like(us) for _ in gusts]
        S, D = torch.empty_like(F), torch.empty_like(F)
        LL = torch.zeros_like(F, dtype=torch.bool)
        st = torch.empty((3, ml, F.shape[2]), device=DEV, dtype=F.dtype)
        air = x["roairn"]
        for m in range(ml):
            sig = ZPI * T["fr"][m]
            xk = x["tfak"][m] if sh else torch.full_like(us, sig * sig / G)
            cm = xk / sig
            constf = row * G / air.clamp(min=1.0) * cm * T["dfim"][m]
            zcn, cnsn = torch.log(xk * z0), sig * cf["betamax"] / kap ** 2 / row * air
            coef, coef5 = -(0.66 * 16 * sig * sig / (G * row)), -(1.2 * 2 * math.sqrt(2 * nu * sig) / row)
            tot_s, tot_d = 0.0, 0.0
            for g in range(2):
                px, py = tx[g] - shelter * xs[g], ty[g] - shelter * ys[g]
                ustp, dirp = (px * px + py * py) ** 0.25, torch.atan2(px, py)
                ucn = ustp * cm
                co = torch.cos(x["th"] - dirp)
                zl = zcn + kap / (ucn + cf["zalp"]) / torch.where(co > 0.01, co, 1.0)
                on = (co > 0.01) & (zl < 0)
                z2x = torch.where(on, zl * zl * co * ucn, 0.0)
                uf = torch.exp(torch.where(on, zl, 0.0)) * z2x * z2x
                LL[m] |= on
                damp = coef5 * air * pvisc * xk + pturb * (coef * air * (temp2 + (0.022 - 0.018 * co) * ustp))
                sl = cnsn * uf
                tot_d = tot_d + 0.5 * (sl + damp)
                sl = sl * F[m]
                xs[g] = xs[g] + (sl * sn).sum(0) * constf
                ys[g] = ys[g] + (sl * cs).sum(0) * constf
                tot_s = tot_s + 0.5 * sl
            D[m], S[m] = tot_d, tot_d * F[m]
            st[0, m], st[1, m], st[2, m] = tot_s.sum(0), (tot_s * sn).sum(0), (tot_s * cs).sum(0)
        return S, D, LL, st

    def _stresso(self, F, st, mij, us, z0):
        x, T, cf = self.x, self.T, self.cfg
        ml = T["ml"]
        m = torch.arange(1, ml + 1, device=DEV)[:, None]
        rw = _t64(T["rhowg"])[:, None] * torch.where((m == mij) & (mij != ml), 0.5, 1.0) * (m <= mij)
        cm = x["tfak"] / x["sig"] if self.c["shallow"] else x["sig"] / G
        px, py = (st[1] * cm * rw).sum(0), (st[2] * cm * rw).sum(0)
        cw = torch.cos(x["th"] - x["udir"]).clamp(min=0.0)
        fm = torch.gather(F, 0, (mij - 1)[None, None].expand(1, F.shape[1], -1))[0]
        t1 = (fm * cw ** 3).sum(0)
        frm = x["fr"][:, 0][mij - 1]
        # high-frequency tail of the stress (Simpson's rule over 19 points)
        kap = 0.40
        x0 = 0.005
        for _ in range(30):
            ff = math.exp(kap / (x0 + cf["zalp"]))
            f = cf["alpha"] * x0 ** 2 * ff - 1.0
            x0 = x0 - f / (cf["alpha"] * ff * (2 * x0 - kap * (x0 / (x0 + cf["zalp"])) ** 2))
        c1 = cf["betamax"] / kap ** 2 / 3.0
        omc = torch.maximum(ZPI * frm, x0 * G / us)
        sq = torch.sqrt(z0 / G)
        zinf = torch.log(omc * sq)
        dz = (-zinf / 18).clamp(min=0.0)
        tw, ust, tau = us * us, us, torch.zeros_like(us)
        for j in range(19):
            y = torch.exp(zinf + j * dz)
            cm1 = y / sq / G
            zl = (torch.log(G * z0) + 2 * torch.log(cm1) + kap / (ust * cm1 + cf["zalp"])).clamp(max=0.0)
            wt = c1 if j in (0, 18) else (4 * c1 if j % 2 else 2 * c1)
            ust = tw.sqrt()
            tau = tau + torch.exp(zl) * zl ** 4 * tw * wt * dz
        hf = T["delth"] * ZPI ** 4 / G * frm ** 5 / G * t1 * tau
        xs = px / 1.225 + hf * torch.sin(x["udir"])
        ys = py / 1.225 + hf * torch.cos(x["udir"])
        return torch.minimum(torch.sqrt(xs * xs + ys * ys), us * us - 1e-5).clamp(min=0.0)

    def _sdissip_ard(self, F, S, D):
        x, T = self.x, self.T
        sig = x["sig"]
        if self.c["shallow"]:
            fac = x["tfak"] ** 3 / ZPI * x["tcg"]
        else:
            k = sig * sig / G
            fac = (k ** 3 * 0.5 / ZPI * G / sig).expand(T["ml"], F.shape[2])
        b = sum(wt * F.roll(-o, 1) for o, wt in T["sat"]) * fac[:, None]
        d0 = (b.amax(1) / 9e-4 - 1).clamp(min=0.0)
        dd = (b / 9e-4 - 1).clamp(min=0.0)
        d = (-2.2e-5 * sig)[:, None] * (0.3 * d0[:, None] ** 2 + 0.7 * dd ** 2)
        return S + d * F, D + d

    def _wavnu2(self, H):
        w0 = self.x["sig"].expand(-1, H.shape[0])
        k = torch.where(w0 < torch.sqrt(G / H), w0 / torch.sqrt(G * H), w0 * w0 / G)
        old = torch.zeros_like(k)
        live = torch.ones_like(k, dtype=torch.bool)
        for _ in range(15):
            dif = (k - old).abs()
            live = live & ~((dif < 1e-7) & (dif / k < 1e-7))
            old = torch.where(live, k, old)
            kh = old * H
            t = torch.tanh(kh)
            ch = torch.cosh(kh.clamp(max=300.0))
            fd = torch.where(kh > 25, G * t, G * t + G * old * H / ch ** 2)
            k = torch.where(live, old - (G * old * t - w0 * w0) / fd, k)
        x = 2 * k * H
        return k, torch.where(x > 25, 0.5 * w0 / k, 0.5 * w0 / k * (1 + x / torch.sinh(x.clamp(max=300.0))))

    def _sinput_st6(self, F, us, depth):
        x, T = self.x, self.T
        nk, kl, n10 = T["ml"], T["kl"], T["nk10"]
        wn, cg = self._wavnu2(depth)
        self.x.update(wn=wn, cg=cg)
        sig, u10, air = x["sig"], x["u10"], x["roairn"]
        cu, su, up = torch.cos(x["udir"]), torch.sin(x["udir"]), 32 * us
        A = F * (cg / (ZPI * sig))[:, None]
        mx = A.amax(1)
        s2 = torch.where(mx < 1e-34, float(kl), (A / torch.where(mx < 1e-34, 1.0, mx)[:, None]).sum(1))
        sqb = torch.sqrt(A.sum(1) * sig * T["delth"] / (s2 * T["delth"]) * wn ** 3)
        ci = wn / sig
        sn, cs = torch.sin(x["th"]), torch.cos(x["th"])
        proj = (up * ci)[:, None] * (cs * cu + sn * su)[None] - 1
        w1, w2 = proj.clamp(min=0.0) ** 2, proj.clamp(max=0.0) ** 2
        gsel = 2.8 - (1 + torch.tanh(10 * sqb[:, None] * torch.where(proj > 0, w1, w2) - 11))
        base = (air / 1000.0 * sig * sqb)[:, None] * gsel
        d1, d2 = torch.where(proj > 0, base * w1, 0.0), torch.where(proj > 0, 0.0, base * 0.09 * w2)
        sd = (d1 * A * sig[:, None] / cg[:, None]).clamp(min=0.0)
        sx, sy = (sd * cs).sum(1) * T["delth"], (sd * sn).sum(1) * T["delth"]
        s10, ds = _t64(T["sig10"])[:, None], _t64(T["ds10"])[:, None]
        r = (s10[nk - 1] / s10[nk:]) ** 2
        sx, sy = torch.cat([sx, sx[-1] * r]), torch.cat([sy, sy[-1] * r])
        c10 = torch.cat([ci, (s10[nk:] * 0.101978).expand(-1, us.shape[0])])
        tot = us * us * air
        vis = torch.minimum(0.95 * tot, (-5e-5 * u10 + 1.1e-3).clamp(min=0.0) * u10 ** 2 * air)
        gro = G * 1000.0
        stress = lambda lf: (gro * (sx * lf * c10 * ds).sum(0), gro * (sy * lf * c10 * ds).sum(0))
        total = lambda a, b: torch.sqrt((vis * cu + a) ** 2 + (vis * su + b) ** 2)
        lf = torch.ones_like(c10)
        tx, ty = stress(lf)
        tau = total(tx, ty)
        err = (tau - tot) / tot
        live = tau > tot
        rt, dr = err / 90, torch.full_like(err, 2.0)
        sgn, over = err >= 0, torch.zeros_like(live)
        for _ in range(80):
            if not bool(live.any()):
                break
            l2 = torch.exp(((1 - up * c10) * rt)).clamp(max=1.0)
            lf = torch.where(live, l2, lf)
            a, b = stress(lf)
            tx, ty = torch.where(live, a, tx), torch.where(live, b, ty)
            err = (total(tx, ty) - tot) / tot
            new = err >= 0
            over = over | (live & (new != sgn))
            sgn = torch.where(live, new, sgn)
            dr = torch.where(live & over, (0.5 * (1 + dr)).clamp(min=1.0001), dr)
            rt = torch.where(live, torch.where(sgn, rt * dr, rt / dr), rt)
            live = live & (err.abs() >= 1.54e-4)
        d = d1 * torch.where(lf[:nk].sum(0) < nk, lf[:nk], 1.0)[:, None]
        D = d - d2
        return D * F, D, d * F > 0, torch.sqrt(tx * tx + ty * ty)

    def _sdissip_st6(self, F, S, D):
        x, T = self.x, self.T
        wn, cg, sig = x["wn"], x["cg"], x["sig"]
        nk, kl = T["ml"], T["kl"]
        et = ZPI * 0.035 ** 2 / (cg * wn ** 3)
        nex4 = ((F.sum(1) * T["delth"] - et).clamp(min=0.0) / et) ** 4
        xfac = (1 - 1 / 1.1) / (1.1 - 1 / 1.1)
        dfii = _t64(T["df"])[:, None] * torch.tensor([1.0] + [xfac] * (nk - 2) + [1.0], device=DEV,
                                                    dtype=torch.float64)[:, None]
        t12 = -(4.75e-6 * x["fr"] * nex4 + 7e-5 * (nex4 * dfii).cumsum(0))
        A = F * (cg / (ZPI * sig))[:, None]
        sa, mx = A.sum(1), A.amax(1)
        s2 = torch.where(mx < 1e-34, float(kl), (A / torch.where(mx < 1e-34, 1.0, mx)[:, None]).sum(1))
        bn = sa * sig * T["delth"] / (s2 * T["delth"]) * wn ** 3
        total = (sa * ZPI * _t64(T["dfim"])[:, None] * sig / cg).sum(0)
        b1 = 0.0041 * 2 * total.sqrt() * torch.gather(wn, 0, sa.argmax(0)[None])[0]
        ab = torch.where(sa > 1e-30, -(2.0 / 3.0 * b1 * sig * bn.sqrt()), 0.0)
        d = (t12 + ab)[:, None]
        return S + d * F, D + d

    def _snonlin(self, F, S, D, ak, depth):
        """Discrete interaction approximation with the spectrum extended below
        by the low-frequency shape and above by an f^-5 tail."""
        T, c = self.T, self.c
        ml, kl = T["ml"], T["kl"]
        enh = torch.ones_like(depth)
        if c["shallow"] and c["isnonlin"] == 0:
            e = (0.75 * depth * ak).clamp(min=0.5)
            enh = 1 + 5.5 / e * (1 - 0.833 * e) * torch.exp(-1.25 * e)
        isp, ism = 2, -4
        first, last = 1 + ism, ml - ism
        fr = lambda m: T["fr"][m - 1] if 1 <= m <= ml else (T["fr"][0] / 1.1 ** (1 - m) if m < 1
                                                             else T["fr"][-1] * 1.1 ** (m - ml))
        ep = lambda y: math.exp(-min(1.25 * y ** 4, 50.0)) * y ** 5
        low = lambda m: ep(1.1 ** (1 - m)) / ep(1.0)
        frh = lambda i: (1.0 / 1.1 ** (i - 1)) ** 5  # FRH(i)
        kfrh = -ism + isp + 2
        a1, b1, a2, b2 = 1 - T["acl1"], T["acl1"], 1 - T["acl2"], T["acl2"]
        S, D = S.clone(), D.clone()

        def turn(kh):
            """Rotations to the two partner directions of both resonant pairs."""
            s = 1 if kh == 0 else -1
            o1, o2 = s * T["rot1"], s * T["rot2"]
            return o1, o1 + s * T["s1"], o2, o2 + s * T["s2"]

        for mc in range(1, last + 1):
            ip, ip1, im, im1 = mc + isp, mc + isp + 1, mc + ism, mc + ism + 1
            wp = (1.25 * fr(mc) - fr(ip)) / (fr(ip1) - fr(ip))
            wp1 = 1 - wp
            if fr(first) >= 0.75 * fr(mc):
                gm, gm1, wm, wm1, none = 1, 1, 0.0, 0.0, True
            else:
                none = False
                wm = (0.75 * fr(mc) - fr(im)) / (fr(im1) - fr(im))
                gm, gm1, wm1 = im, im1, 1 - wm
                if im < first:
                    gm, wm1 = 1, 0.0
            fic, fp, fp1, fm, fm1 = 1.0, 1.0, 1.0, 1.0, 1.0
            ic, jp, jp1, jm, jm1 = mc, ip, ip1, gm, gm1
            if jm < 1:
                fm, jm = low(gm), 1
                if jm1 < 1:
                    fm1, jm1 = low(gm1), 1
            if jp1 > ml:
                fp1, jp1 = frh(min(ip1 - ml + 1, kfrh)), ml
                if jp > ml:
                    fp, jp = frh(ip - ml + 1), ml
                    if ic > ml:
                        fic, ic = frh(mc - ml + 1), ml
                        if jm1 > ml:
                            fm1, jm1 = frh(gm1 - ml + 1), ml
            if c["shallow"] and c["isnonlin"] != 0:
                enh = self._transf(mc, depth)
            ft = 3000.0 * fr(mc) ** 11 * enh
            tm, tm1 = (mc + ism, mc + ism + 1) if not none else (1, 1)
            if not none and im < first:
                tm = 1
            low_regime = mc <= -first + 1
            high = mc >= ml - kfrh + (-first + 1) and not low_regime
            fij = F[ic - 1] * fic
            for kh in range(2):
                o1, o11, o2, o21 = turn(kh)
                at = lambda row, o: F[row - 1].roll(-o, 0)
                sap = T["dal1"] * (wp1 * fp * (a1 * at(jp, o1) + b1 * at(jp, o11))
                                   + wp * fp1 * (a1 * at(jp1, o1) + b1 * at(jp1, o11)))
                sam = T["dal2"] * (wm1 * fm * (a2 * at(jm, o2) + b2 * at(jm, o21))
                                   + wm * fm1 * (a2 * at(jm1, o2) + b2 * at(jm1, o21)))
                fad1 = fij * (sap + sam)
                fad2 = fad1 - 2 * sap * sam
                fad1 = fad1 + fad2
                ad, delad = fad2 * ft * fij, fad1 * ft
                delap = (fij - 2 * sam) * T["dal1"] * ft * fij
                delam = (fij - 2 * sap) * T["dal2"] * ft * fij
                if mc <= ml:
                    S[mc - 1] -= 2 * ad
                    D[mc - 1] -= 2 * delad
                def put(row, o, weight, dd):
                    if 1 <= row <= ml:
                        S[row - 1] += (weight * ad).roll(o, 0)
                        D[row - 1] += (weight * weight * dd).roll(o, 0)
                if not low_regime:
                    put(tm, o2, wm1 * a2, delam)
                    put(tm, o21, wm1 * b2, delam)
                if not (low_regime and tm1 < 1):
                    put(tm1, o2, wm * a2, delam)
                    put(tm1, o21, wm * b2, delam)
                put(ip, o1, wp1 * a1, delap)
                put(ip, o11, wp1 * b1, delap)
                put(ip1, o1, wp * a1, delap)
                put(ip1, o11, wp * b1, delap)
        return S, D

    def _transf(self, mc, depth):
        """Depth factor of the quadruplets at frequency index mc."""
        T = self.T
        fr = T["fr"][mc - 1] if mc <= T["ml"] else T["fr"][-1] * 1.1 ** (mc - T["ml"])
        om = ZPI * fr
        k = torch.maximum(torch.full_like(depth, om * om / (4 * G)), om / (2 * torch.sqrt(G * depth)))
        for _ in range(30):
            bo = (depth * k).clamp(max=40.0)
            t = G * k * torch.tanh(bo)
            st = t.sqrt()
            k = torch.where(depth * k > 40.0, om * om / G,
                            k + (om - st) * st * 2 / (t / k + G * bo / torch.cosh(bo) ** 2))
        x = (k * depth).clamp(max=40.0)
        t0 = torch.tanh(x)
        c0 = torch.sqrt(G * k * t0) / k
        vg = 0.5 * c0 * (1 + 2 * x / torch.sinh(2 * x))
        t2 = t0 * t0
        dvg = (t0 - x * (1 - t2)) ** 2 + 4 * x ** 2 * t2 * (1 - t2)
        x1 = (9 * t2 * t2 - 10 * t2 + 9) / (8 * t0 ** 3)
        x2 = ((2 * vg - 0.5 * c0) ** 2 / (G * depth - vg * vg) + 1) / x
        r = ((x1 - x2) ** 2 / (dvg * t0 ** 8)).clamp(max=10.0)
        return torch.where((depth < 999.0) & (k * depth <= 40.0), r, 1.0)

    # ---- integrated output --------------------------------------------------
    def output(self, F, ustar, z0):
        T, w, c = self.T, self.w, self.c
        u10, udir, tauw, depth = (_t64(w[q]) for q in ("u10", "udir", "tauw", "depth"))
        deg = 180.0 / PI
        B = torch.zeros((40, w["n"]), device=DEV, dtype=torch.float64)
        dfim, fr = _t64(T["dfim"])[:, None], _t64(T["fr"])[:, None]
        df, delth = _t64(T["df"])[:, None], T["delth"]
        sn, cs = _t64(np.sin(T["th"]))[:, None], _t64(np.cos(T["th"]))[:, None]

        def integrals(F):
            t = F.sum(1)
            e = ((t * dfim).sum(0) + T["mo_tail"] * t[-1]).clamp(min=1e-12)
            fm = e / ((t * dfim / fr).sum(0) + T["mm1_tail"] * t[-1]).clamp(min=1e-12)
            m1 = (t * df * fr * delth).sum(0) + T["mp1_tail"] * t[-1]
            m2 = (t * df * fr ** 2 * delth).sum(0) + T["mp2_tail"] * t[-1]
            ok = e > 1e-12
            ip = t.argmax(0)
            d = (F * dfim[:, None]).sum(0)
            si, ci, sp = (sn * d).sum(0), (cs * d).sum(0), d.sum(0)
            thq = torch.atan2(si, torch.where(ci == 0, 0.1e-30, ci))
            thq = torch.where(thq < 0, thq + ZPI, thq)
            thq = torch.where(thq > ZPI - 0.001, 0.0, thq)
            lim = lambda v: torch.where(v.abs() < 1e-16, torch.copysign(torch.full_like(v, 1e-16), v), v)
            spr = 2 * (1 - torch.sqrt(lim(si) ** 2 + lim(ci) ** 2) / lim(sp))
            spr = torch.where(spr <= 0, 1.1754943508222875e-38, spr.clamp(min=0).sqrt())
            return [4 * e.sqrt(), torch.where(ip == 0, 1.0, 1 / fr[:, 0][ip]), 1 / fm, torch.where(ok, e / m1, 1.0),
                    torch.where(ok, torch.sqrt(e / m2), 1.0), thq * deg, spr * deg]

        B[0], B[1], B[2] = u10, deg * udir, ustar
        tau = ustar ** 2 + 1e-4
        B[3], B[15] = tau / (u10 ** 2 + 0.01), tauw / (tau * 1.225)
        B[4] = G * z0 / (ustar ** 2).clamp(min=1e-6)
        B[5] = depth if c["shallow"] else 999.0
        B[31] = z0
        t = F.sum(1)
        if c["shallow"]:
            B[39] = 1e-33 + (dfim * self.tfak[:, self.iind] ** 2 * t).sum(0)
        else:
            B[39] = 1e-33 + (dfim * (ZPI * fr) ** 4 / G ** 2 * t).sum(0)
        for row, v in zip(range(8, 15), integrals(F)):
            B[row] = v
        th, cph = _t64(T["th"])[None, :, None], (G / (ZPI * fr))[:, None]
        swell = 28.0 / cph * 1.2 * ustar * torch.cos(th - udir) < 1.0
        sw = torch.where(swell, F.clamp(min=1e-33), 0.0)
        for row, v in zip(range(16, 23), integrals(torch.where(swell, F - sw, F))):
            B[row] = v
        for row, v in zip(range(24, 31), integrals(sw)):
            B[row] = v
        return B


def _exact_step(c, w, props, source):
    x = _Exact64(c, w)
    f = _spectrum(c, w, DEV, torch.float32).double()
    tauw = _t64(w["tauw"])
    if props:
        cnt = x.counter()
        for _ in range(props):
            f = x.propagate(f, cnt)
    out = {}
    if source:
        f, tauw, out["ustar"], out["z0"] = x.implsch(f, tauw)
        out["tauw"] = tauw
    full = torch.zeros((c["ml"], c["kl"], w["n"] + c["pad"]), device=DEV, dtype=torch.float64)
    full[:, :, :w["n"]] = f
    out["f"] = full
    return out


def exact(case, seed):
    c = case
    nprop = c["idelt"] // c["idelpro"]
    if c["kind"] == "window":
        return None  # derivatives of the whole window: no plain evaluation within the time
    if c["kind"] == "ensemble":
        outs = []
        for k in range(c["members"]):
            mc = _member(c, k)
            o = _exact_step(mc, _inputs(mc, seed + 1000 * k), nprop, True)
            outs.append(dict(f=o["f"], tauw=o["tauw"], ustar=o["ustar"]))
        return outs
    w = _inputs(c, seed)
    if c["kind"] == "output":
        us = torch.tensor(w["u10"] * np.sqrt(1e-3 * (0.8 + 0.08 * w["u10"])), device=DEV).float()
        z0 = us ** 2 * (0.012 / G)
        f = _spectrum(c, w, DEV, torch.float32).double()
        return dict(block=_Exact64(c, w).output(f, us.double(), z0.double()))
    if c["kind"] == "hosted":
        c = dict(c, pad=0)
    return _exact_step(c, w, {"implsch": 0, "propags": 1}.get(c["kind"], nprop), c["kind"] != "propags")
