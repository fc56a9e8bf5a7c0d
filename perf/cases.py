"""Performance cases: the framework's work through its public entry points.

A case is a dict of plain values.  `listed()` gives the fixed set, `draw()` one
more of the same ranges, `prepare()` what a caller holds before the call,
`run()` one pass, `work()` the bytes and operations the pass cannot do without
and `exact()` the pass's outputs in 64 bits from plain torch and numpy.

Kinds of case
  engine  batched number counts (and stacked miscentred Delta Sigma) of one
          y3b_engine call: `api` "device" (buffers resident in HBM), "host"
          (pinned host buffers through the C ABI) or "python" (Engine.eval)
  serve   a burst of requests through the request server
  module  the CosmoSIS module chain of one sample: sel_function, then the
          number-count and shear operators on its table
  prj     projection shear of one sample
  bsel    selection-bias operators of a batch of samples
"""
import ctypes
import math

import numpy as np
import torch

from y3_cluster_cpp_b200 import _capi, prj_params
from y3_cluster_cpp_b200 import engine as E
from y3_cluster_cpp_b200 import serve

DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")
F64 = torch.float64
RHO_CRIT = 2.77533742639e11
C_OVER_H0 = 2997.92458
LAM_EDGES = (20.0, 30.0, 45.0, 60.0, 200.0)
ZOB_EDGES = (0.20, 0.35, 0.50, 0.65)
LOB = (25.0, 37.5, 52.5, 130.0)
LNM = (math.log(1e13), math.log(10 ** 15.5))
ZT = (0.1, 0.8)
LAM_T = (1.0, 1000.0)
SZ0 = 0.01
H0 = 0.7
NODES = ("n_m", "n_z", "n_t", "n_o", "n_zo")
DENSITY = {1: (64, 32, 64, 64, 16), 2: (128, 64, 128, 128, 32), 4: (256, 128, 256, 256, 64)}


# ---------------------------------------------------------------------------
# The cases.
def _engine(name, api, precision, n, nodes, radii=0, hmf_fp32=False, loglike=False):
    c = dict(name=name, kind="engine", api=api, precision=precision, n=n, radii=radii,
             hmf_fp32=hmf_fp32, loglike=loglike)
    c["mixed_density"] = nodes is None
    c.update(zip(NODES, nodes or DENSITY[4]))
    return c


def listed():
    return [
        # one likelihood point of a running chain, the default 1x nodes: latency
        _engine("chain_point_1x", "python", "mixed", 1, DENSITY[1]),
        # an ensemble sampler's step, host tables with the FP32 HMF grid, odd node counts
        _engine("ensemble_host_ragged", "host", "mixed", 777, (150, 80, 200, 96, 24),
                hmf_fp32=True),
        # a large batch at 4x nodes, resident in HBM
        _engine("batch_counts_4x", "device", "mixed", 2048, DENSITY[4], hmf_fp32=True),
        # walkers of three node densities with counts and Delta Sigma in one call
        _engine("walkers_uneven_shear", "device", "mixed", 256, None, radii=15),
        # counts, Delta Sigma and the fused likelihood at 1x nodes
        _engine("likelihood_1x", "device", "mixed", 2048, DENSITY[1], radii=15, loglike=True),
        # the FP64 form: reference-grade counts at 4x nodes
        _engine("fp64_counts_4x", "device", "fp64", 48, DENSITY[4]),
        # the FP64 form with Delta Sigma through host buffers
        _engine("fp64_shear_host", "host", "fp64", 12, (64, 32, 64, 64, 16), radii=15),
        # a burst of requests of 1..64 points from several samplers
        dict(name="serve_burst", kind="serve", requests=24, max_points=64),
        # one CosmoSIS sample of the module path at its default node counts
        dict(name="module_sample", kind="module", mor="hod", tab_m=192, tab_z=64, n_q=32,
             n_lnm=96, n_z=64, radii=15),
        # one sample of the projection shear: 12 slices x 10 radii
        dict(name="prj_sample", kind="prj", radii=10, n_lnm=24, n_per_seg=10, n_zring=20,
             n_zouter=20),
        # selection-bias operators: one sample of a chain, and a batch of walkers
        dict(name="bsel_sample", kind="bsel", n=1, n_lt=60, n_zring=20, n_zouter=30, n_lnm=24,
             n_theta=10, n_zt_ref=80),
        dict(name="bsel_batch", kind="bsel", n=192, n_lt=60, n_zring=20, n_zouter=30, n_lnm=24,
             n_theta=10, n_zt_ref=80),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("engine", "serve", "module", "prj", "bsel"), (12, 2, 2, 2, 3))[0]
    if kind == "serve":
        return dict(kind=kind, requests=rng.randint(6, 24), max_points=_log_int(rng, 4, 64))
    if kind == "module":
        return dict(kind=kind, mor=rng.choice(("hod", "lognormal")), tab_m=rng.randint(96, 192),
                    tab_z=rng.randint(32, 64), n_q=rng.randint(16, 32), n_lnm=rng.randint(48, 96),
                    n_z=rng.randint(32, 64), radii=rng.randint(5, 15))
    if kind == "prj":
        return dict(kind=kind, radii=rng.randint(3, 10), n_lnm=rng.randint(12, 24),
                    n_per_seg=rng.randint(6, 10), n_zring=rng.randint(10, 20),
                    n_zouter=rng.randint(10, 20))
    if kind == "bsel":
        return dict(kind=kind, n=_log_int(rng, 1, 192), n_lt=rng.randint(30, 60),
                    n_zring=rng.randint(10, 20), n_zouter=rng.randint(15, 30),
                    n_lnm=rng.randint(12, 24), n_theta=rng.randint(6, 10),
                    n_zt_ref=rng.randint(40, 80))
    fp64 = rng.random() < 0.3
    radii = rng.choice((0, 0, rng.randint(1, 15)))
    n = _log_int(rng, 1, 2048)
    if fp64:
        n = _log_int(rng, 1, 12 if radii else 48)
    elif radii:
        n = min(n, 1024)
    if rng.random() < 0.2 and n >= 3 and not (fp64 and radii):
        nodes = None
    else:
        top = 64 if fp64 and radii else 256
        nodes = (_log_int(rng, 32, top), 16 * rng.randint(1, 2 if top == 64 else 8),
                 _log_int(rng, 32, top), _log_int(rng, 32, 256), _log_int(rng, 8, 64))
    c = _engine("", rng.choice(("device", "host", "python")) if n <= 64
                else rng.choice(("device", "host")), "fp64" if fp64 else "mixed", n, nodes, radii,
                hmf_fp32=not fp64 and rng.random() < 0.5)
    c.pop("name")
    return c


# ---------------------------------------------------------------------------
# Synthetic inputs, batched over walkers (float64 tensors on DEV).
def _t(x):
    return torch.as_tensor(x, dtype=F64, device=DEV)


def _growth(z, om):
    def g(x):
        a3 = (1 + x) ** 3
        e2 = om * a3 + (1 - om)
        omz, olz = om * a3 / e2, (1 - om) / e2
        return 2.5 * omz / (omz ** (4 / 7) - olz + (1 + omz / 2) * (1 + olz / 70))

    return g(z) / g(torch.zeros_like(z)) / (1 + z)


def _walkers(n, seed, sci=True):
    """Parameters and tables of n walkers: Omega_m U[0.2, 0.4], sigma8
    U[0.7, 0.9], A, B and sigma_int within 20 %."""
    r = np.random.default_rng(seed)
    u = r.uniform(size=(n, 5))
    w = dict(om=0.2 + 0.2 * u[:, 0], s8=0.7 + 0.2 * u[:, 1], A=3.2 * (0.8 + 0.4 * u[:, 2]),
             B=0.9 * (0.8 + 0.4 * u[:, 3]), sigma=0.2 * (0.8 + 0.4 * u[:, 4]))
    om, s8 = _t(w["om"])[:, None], _t(w["s8"])[:, None, None]
    M = _t(np.logspace(13, 15.5, 100))
    hz = _t(np.linspace(ZT[0], ZT[1], 50))
    D = _growth(hz[None, :], om)
    sig = s8 * (M / 2e14) ** -0.2 * D[:, :, None]
    zp = 1 + hz[None, :, None]
    al = 10 ** (-((0.75 / math.log10(200 / 75.0)) ** 1.2))
    f = 0.186 * zp ** -0.14 * (sig / (2.57 * zp ** -al)) ** (-1.47 * zp ** -0.06) \
        * torch.exp(-1.19 / sig ** 2)
    w["hmf_m_h"] = M / om
    w["hmf_z"] = hz
    w["dn"] = f * (om * RHO_CRIT)[:, :, None] / M * 0.2
    nd, sub = 200, 16
    zz = _t(np.linspace(0.0, 2.0, (nd - 1) * sub + 1))
    ie = 1.0 / torch.sqrt(om * (1 + zz) ** 3 + (1 - om))
    h = float(zz[1])
    two = torch.cumsum(h / 3 * (ie[:, :-2:2] + 4 * ie[:, 1:-1:2] + ie[:, 2::2]), 1)
    chi = torch.cat([torch.zeros(n, 1, dtype=F64, device=DEV), two], 1)[:, :: sub // 2]
    w["dist_z"] = _t(np.linspace(0.0, 2.0, nd))
    w["dist_dc"] = chi * C_OVER_H0 / H0
    w["dist_da"] = w["dist_dc"] / (1 + w["dist_z"])
    if sci:
        zl, zs = _t(np.linspace(0.05, 0.85, 64)), _t(np.linspace(0.01, 2.0, 200))
        p = torch.exp(-0.5 * ((zs - 0.9) / 0.3) ** 2)
        p = p / torch.trapezoid(p, zs)
        dl, ds = _lin(w["dist_z"], w["dist_da"], zl), _lin(w["dist_z"], w["dist_da"], zs)
        k = 4 * math.pi * 4.51710305e-48 / 9.71561189e-15 ** 2
        dls = ds[:, None, :] - ((1 + zl)[:, None] / (1 + zs)) * dl[:, :, None]
        w["sci_z"] = zl
        w["sci_val"] = torch.trapezoid((p * k * dl[:, :, None] * dls / ds[:, None, :]).clamp(min=0),
                                       zs) * H0
    return w


def _halo_tables(w, n_r):
    """Halo bias and nonlinear correlation function of each walker."""
    om, s8 = _t(w["om"])[:, None], _t(w["s8"])[:, None, None]
    lnM, z = _t(np.linspace(math.log(1e12), math.log(1e16), 60)), _t(np.linspace(0.0, 1.2, 40))
    D = _growth(z[None, :], om)[:, :, None]
    nu = 1.686 / (s8 * (torch.exp(lnM) / 2e14) ** -0.2 * D)
    r = _t(np.logspace(-2, math.log10(5000.0), n_r))
    xi = (r / 5.0) ** -1.8 * torch.exp(-r / 200.0) * D ** 2
    return dict(halo_lnM=lnM, halo_z=z, bias=1.0 + (nu * nu - 1.0) / 1.686, xi_r=r, xi_z=z,
                xi_nl=xi)


def _plob():
    """P(lam_o | lam_t): Gaussian of width 0.1 lam_t with a projection tail of
    weight 0.1, constant in z (rows a_tau, b_tau, a_mu, b_mu, a_sig, b_sig,
    a_fprj, b_fprj)."""
    v = np.array([0.672770912, 1.95006009, 0.0, 1.0, 1.0, 0.1, 0.0, 0.1])
    return np.array([0.0, 2.0]), np.repeat(v[:, None], 2, 1)


def _grid(nodes):
    g = dict(zip(NODES, nodes))
    g.update(lnm_lo=LNM[0], lnm_hi=LNM[1], zt_lo=ZT[0], zt_hi=ZT[1], lam_t_lo=LAM_T[0],
             lam_t_hi=LAM_T[1], lam_edges=LAM_EDGES, zob_edges=ZOB_EDGES, sz0=SZ0)
    return g


def _radii(n):
    return np.logspace(math.log10(0.1), math.log10(30.0), n)


def _shear_opts(n):
    return dict(R=_radii(n), f_mis=0.2, tau_mis=0.17, lob_centers=LOB, c0=5.0, c_slope=-0.1,
                c_pivot=1e14, n_theta=64, n_s=128, s_max=20.0)


def _node_sets(case):
    return [DENSITY[d] for d in (1, 2, 4)] if case.get("mixed_density") \
        else [tuple(case[k] for k in NODES)]


def _grid_index(n, n_grids):
    return np.arange(n) * n_grids // max(n, 1)


def _points(w, idx):
    """y3b_point records of the walkers."""
    n = len(idx)
    p = np.zeros(n, dtype=[("v", "f8", 12), ("grid", "i4"), ("reserved", "i4")])
    v = p["v"]
    v[:, 0], v[:, 1], v[:, 3], v[:, 6] = w["om"], 1.0 - w["om"], H0, 1.0
    v[:, 7], v[:, 8], v[:, 9], v[:, 10], v[:, 11] = w["A"], w["B"], 0.5, w["sigma"], 3e14
    p["grid"] = idx
    return np.frombuffer(p.tobytes(), dtype=np.uint8).copy()


def _pack(eng, w, n):
    """Packed per-point tables of the engine [n, stride]."""
    buf = torch.zeros((n, eng.stride), dtype=F64, device=DEV)
    vals = (w["hmf_m_h"], w["hmf_z"], w["dn"].reshape(n, -1), w["dist_z"], w["dist_da"],
            w.get("sci_z"), w.get("sci_val"))
    for o, v, m in zip(eng.offsets, vals, (100, 50, 5000, 200, 200, 64, 64)):
        if v is None or eng.shapes[3] == 0 and m == 64:
            continue
        if eng.hmf_fp32 and m == 5000:
            buf[:, o:o + 2500] = v.float().contiguous().view(F64)
        else:
            buf[:, o:o + m] = v
    return buf


class _Walker:
    """A sampler point as Engine.eval reads it."""

    def __init__(self, w, i, grid):
        self.om, self.h0, self.C, self.Mpiv = float(w["om"][i]), H0, 0.5, 3e14
        self.A, self.B, self.sigma = (float(w[k][i]) for k in ("A", "B", "sigma"))
        self.grid_index = int(grid)


def _data_vector(case, seed):
    """Mock counts and shear near a walker's, with 10 % diagonal errors."""
    w = _walkers(1, seed + 501)
    counts, shear = _engine_exact(w, [DENSITY[1]], np.zeros(1, int), case["radii"])
    r = np.random.default_rng(seed + 502)
    d = counts[0].cpu().numpy() * (1 + 0.05 * r.standard_normal(12))
    s = (shear[0] / counts[0][:, None]).cpu().numpy()
    s = s * (1 + 0.05 * r.standard_normal(s.shape))
    return d, 1.0 / (0.1 * d) ** 2, s.ravel(), 1.0 / (0.1 * s.ravel()) ** 2


# ---------------------------------------------------------------------------
# State and pass.
def _prepare_engine(case, seed):
    n = case["n"]
    sets = _node_sets(case)
    idx = _grid_index(n, len(sets))
    w = _walkers(n, seed, sci=case["radii"] > 0)
    eng = E.Engine([_grid(s) for s in sets], 100, 50, 200, _plob(), max_points=n,
                   n_sci=64 if case["radii"] else 0,
                   shear=_shear_opts(case["radii"]) if case["radii"] else None,
                   hmf_fp32=case["hmf_fp32"])
    tab, pts = _pack(eng, w, n), torch.from_numpy(_points(w, idx))
    s = dict(case=case, eng=eng, n=n, prec=E.MIXED if case["precision"] == "mixed" else E.FP64)
    nB, nR = eng.n_bins, eng.n_R
    if case["api"] == "device":
        s["pts"], s["tab"] = pts.to(DEV), tab
        s["counts"] = torch.empty((n, nB), dtype=F64, device=DEV)
        s["shear"] = torch.empty((n, nB, nR), dtype=F64, device=DEV) if nR else None
    elif case["api"] == "host":
        pin = dict(pin_memory=True)
        s["pts"], s["tab"] = pts.pin_memory(), torch.empty(tab.shape, dtype=F64, **pin).copy_(tab)
        s["counts"] = torch.empty((n, nB), dtype=F64, **pin)
        s["shear"] = torch.empty((n, nB, nR), dtype=F64, **pin) if nR else None
    else:
        s["pts"] = [_Walker(w, i, idx[i]) for i in range(n)]
        s["tab"] = tab.cpu().numpy()
    if case["loglike"]:
        eng.set_likelihood(E.LikelihoodSpec(*_data_vector(case, seed)))
    return s


def _ptr(t, kind=ctypes.c_double):
    return ctypes.cast(t.data_ptr() if t is not None else None, ctypes.POINTER(kind))


def _run_engine(s):
    eng, n, c = s["eng"], s["n"], s["case"]
    if c["api"] == "python":
        r = eng.eval(s["pts"], s["prec"], tables=s["tab"], grid_of=lambda p: p.grid_index)
        return [r["counts"], r["shear"]] if "shear" in r else [r["counts"]]
    if c["api"] == "host":
        E.check(E.lib().y3b_engine_eval(eng.handle, s["prec"], n, _ptr(s["pts"], _capi.Point),
                                        *(_ptr(s[k]) for k in ("tab", "counts", "shear"))))
    else:
        eng.eval_device(s["prec"], n, s["pts"].data_ptr(), s["tab"].data_ptr(),
                        s["counts"].data_ptr(), s["shear"].data_ptr() if eng.n_R else 0)
    out = [s["counts"], s["shear"]] if eng.n_R else [s["counts"]]
    if c["loglike"]:
        out.append(eng.loglike(n))
    return out


def _request_sizes(case):
    r = np.random.default_rng(7)
    return np.rint(np.exp(r.uniform(0, math.log(case["max_points"]), case["requests"]))).astype(int)


def _prepare_serve(case, seed):
    sizes = _request_sizes(case)
    n = int(sizes.sum())
    w = _walkers(n, seed, sci=False)
    idx = np.arange(n) % 3
    eng = E.Engine([_grid(DENSITY[d]) for d in (1, 2, 4)], 100, 50, 200, _plob(),
                   max_points=2048, hmf_fp32=True)
    tab = torch.empty((n, eng.stride), dtype=F64, pin_memory=True).copy_(_pack(eng, w, n)).numpy()
    rec, reqs, o = _points(w, idx), [], 0
    size = ctypes.sizeof(_capi.Point)
    for m in sizes:
        pts = (_capi.Point * int(m)).from_buffer_copy(rec[o * size:(o + m) * size].tobytes())
        reqs.append((pts, tab[o:o + m]))
        o += m
    srv = serve.Server(eng, pool_points=4096, max_batch=2048)
    return dict(case=case, srv=srv, reqs=reqs)


def _run_serve(s):
    tickets = [s["srv"].submit(*r) for r in s["reqs"]]
    return [s["srv"].wait(t)["counts"] for t in tickets]


def _module_inputs(case, seed):
    w = _walkers(1, seed)
    r = np.random.default_rng(seed + 11)
    tab = {k: w[k].cpu().numpy() for k in ("hmf_z", "dist_z", "sci_z")}
    for k, s in (("hmf_m_h", "hmf_m_h"), ("dndlnmh", "dn"), ("dist_da", "dist_da"),
                 ("sci_val", "sci_val")):
        tab[k] = w[s][0].cpu().numpy()
    i, j = np.tile(np.arange(4), 3), np.repeat(np.arange(3), 4)
    cfg = dict(lam_min=np.array(LAM_EDGES)[i], lam_max=np.array(LAM_EDGES)[i + 1],
               zob_min=np.array(ZOB_EDGES)[j], zob_max=np.array(ZOB_EDGES)[j + 1],
               sigma_z=np.full(12, 0.03), zt_low=0.05, zt_high=0.8, lnm_low=29.9336, lnm_high=36.73,
               n_lnm=case["tab_m"], n_z=case["tab_z"], n_q=case["n_q"])
    if case["mor"] == "hod":
        kind, mor = 0, [11.4 + 0.3 * r.uniform(), 12.7, 0.86, 0.1 * r.uniform(), 0.18, 0.45]
    else:
        kind, mor = 1, [float(w["A"][0]), float(w["B"][0]), 0.5, float(w["sigma"][0]), 3e14, 1.0,
                        1000.0]
    om = float(w["om"][0])
    lnM, rs = np.linspace(math.log(1e13), math.log(10 ** 15.9), 60), np.logspace(-2, 2, 80)
    scale = np.cbrt(3 * np.exp(lnM) / (800 * math.pi * RHO_CRIT * om)) / 5.0
    x = _t(rs[None, :] / scale[:, None])
    dc = (200.0 * 125.0 / 3.0) / (math.log(6.0) - 5.0 / 6.0)
    halo = dict(r_sigma=rs, lnM=lnM,
                dSigma_nfw=(2 * scale[:, None] * dc * RHO_CRIT * om * 1e-12)
                * _dsigma(x).cpu().numpy())
    nR = case["radii"]
    return dict(cz=E.cosmo(om, H0), om=om, tab=tab, cfg=cfg, kind=kind, mor=mor,
                plob=prj_params.default_table(), halo=halo, bins=np.repeat(np.arange(12), nR),
                r=np.tile(_radii(nR), 12))


def _prepare_module(case, seed):
    s = _module_inputs(case, seed)
    nodes = dict(n_lnm=case["n_lnm"], n_z=case["n_z"])
    s.update(case=case, nc=E.SelGL(**nodes), sh=E.SelGL(**nodes))
    return s


def _run_module(s):
    sel = E.sel_function(s["cfg"], s["kind"], s["mor"], *s["plob"])
    counts = s["nc"].build(s["cz"], s["tab"], sel).counts(np.arange(12))
    shear = s["sh"].build(s["cz"], s["tab"], sel, include_sci=True).shear(s["bins"], s["r"],
                                                                        s["halo"])
    return [sel[2], counts, shear]


def _sample_tables(w, hal, i):
    t = dict(hmf_m_h=w["hmf_m_h"][i], hmf_z=w["hmf_z"], dndlnmh=w["dn"][i], dist_z=w["dist_z"],
             dist_da=w["dist_da"][i])
    if "sci_z" in w:
        t.update(sci_z=w["sci_z"], sci_val=w["sci_val"][i])
    p = dict(dist_dc=w["dist_dc"][i], bias=hal["bias"][i], xi_nl=hal["xi_nl"][i],
             **{k: hal[k] for k in ("halo_lnM", "halo_z", "xi_r", "xi_z")})
    return tuple({k: v.cpu().numpy() for k, v in d.items()} for d in (t, p))


def _prj_inputs(case, seed):
    w = _walkers(1, seed)
    t, p = _sample_tables(w, _halo_tables(w, 200), 0)
    zob = np.array([0.275, 0.425, 0.575])
    p.update(bsel_lob=np.array(LOB), bsel_zob=zob,
             b_small=(1.0 + 0.1 * np.arange(4)[None, :] + 0.2 * zob[:, None]).ravel(),
             b_large=(2.0 + 0.3 * np.arange(4)[None, :] + 0.5 * zob[:, None]).ravel())
    nR = case["radii"]
    R = np.logspace(math.log10(0.2), math.log10(5.0), nR)
    grid = dict(lambda_bin=np.repeat(np.tile(np.arange(4), 3), nR),
                zo_low=np.repeat(np.repeat(ZOB_EDGES[:3], 4), nR),
                zo_high=np.repeat(np.repeat(ZOB_EDGES[1:], 4), nR), radii=np.tile(R, 12))
    return float(w["om"][0]), t, p, grid


def _prepare_prj(case, seed):
    om, t, p, grid = _prj_inputs(case, seed)
    h = E.PrjShear(grid, **{k: case[k] for k in ("n_lnm", "n_per_seg", "n_zring", "n_zouter")})
    return dict(case=case, h=h, cz=E.cosmo(om, H0), t=t, p=p)


def _bsel_inputs(case, seed):
    n = case["n"]
    w = _walkers(n, seed, sci=False)
    hal = _halo_tables(w, 120)
    r = np.random.default_rng(seed + 13)
    hod = np.stack([11.7 + 0.1 * r.uniform(-1, 1, n), 12.9 + 0.1 * r.uniform(-1, 1, n),
                    0.8 + 0.1 * r.uniform(size=n), 0.2 + 0.1 * r.uniform(-1, 1, n),
                    0.15 + 0.1 * r.uniform(size=n)], 1)
    return w, hal, hod


def _prepare_bsel(case, seed):
    w, hal, hod = _bsel_inputs(case, seed)
    keys = ("log10_Mmin", "log10_M1", "alpha", "epsilon", "sigma_lambda")
    samples = []
    for i in range(case["n"]):
        t, p = _sample_tables(w, hal, i)
        samples.append((E.cosmo(float(w["om"][i]), H0), t, p, dict(zip(keys, hod[i]))))
    grid = dict(zo_low=np.repeat(ZOB_EDGES[:3], 4), zo_high=np.repeat(ZOB_EDGES[1:], 4),
                lambda_bin=np.tile(np.arange(4), 3))
    h = E.BselMarg(grid, *LNM, max_samples=case["n"],
                   **{k: case[k] for k in ("n_lt", "n_zring", "n_zouter", "n_lnm", "n_theta",
                                           "n_zt_ref")})
    return dict(case=case, h=h, samples=samples)


def prepare(case, seed):
    return {"engine": _prepare_engine, "serve": _prepare_serve, "module": _prepare_module,
            "prj": _prepare_prj, "bsel": _prepare_bsel}[case["kind"]](case, seed)


def run(state):
    kind = state["case"]["kind"]
    if kind == "engine":
        return _run_engine(state)
    if kind == "serve":
        return _run_serve(state)
    if kind == "module":
        return _run_module(state)
    if kind == "prj":
        return state["h"].eval(state["cz"], state["t"], state["p"])
    return state["h"].eval(state["samples"])


def work(case):
    """Each input read and each output written once, and the multiply-adds of
    the path's sums (a quadrature node's profile counted as one)."""
    kind = case["kind"]
    if kind in ("engine", "serve"):
        if kind == "serve":
            n, nR, nodes = int(_request_sizes(case).sum()), 0, [DENSITY[d] for d in (1, 2, 4)]
            idx, dn = np.arange(n) % 3, 4
        else:
            n, nR, nodes = case["n"], case["radii"], _node_sets(case)
            idx, dn = _grid_index(n, len(nodes)), 4 if case["hmf_fp32"] else 8
        per = 5000 * dn + 8 * (100 + 50 + 400 + (128 if nR else 0)) + 104 + 8 * 12 * (1 + nR)
        flops = sum(2.0 * nodes[g][0] * 4 * nodes[g][1] * nodes[g][2] + 24.0 * nR * nodes[g][0]
                    for g in idx)
        return dict(bytes=float(n * per), flops=flops)
    tables = 8.0 * (100 + 50 + 5000 + 3 * 200)
    if kind == "module":
        cells, nR = case["tab_m"] * case["tab_z"], case["radii"]
        return dict(bytes=tables + 8.0 * (12 * cells + 60 * 80 + 12 * (1 + nR)),
                    flops=2.0 * cells * case["n_q"] * 4 + 24.0 * 2 * case["n_lnm"] * case["n_z"]
                    + 2.0 * 4 * nR * case["n_lnm"] * 64 * 128)
    if kind == "prj":
        nR = case["radii"]
        nth, nz = case["n_per_seg"] * (nR + 4), case["n_zring"] + 2 * case["n_zouter"]
        return dict(bytes=tables + 8.0 * (2400 + 8000 + 12 * nR * 9),
                    flops=12.0 * (2 * nth * nz + nR * nth * case["n_lnm"] * (2 * 256 + 4)))
    n, nz = case["n"], case["n_zring"] + 2 * case["n_zouter"]
    return dict(bytes=n * (tables + 8.0 * (2400 + 120 * 40 + 36)),
                flops=12.0 * n * nz * case["n_lt"] * (4 * case["n_lnm"] + 4 * case["n_theta"]))


# ---------------------------------------------------------------------------
# The same quantities in 64 bits.
def _gl(a, b, n):
    x, w = np.polynomial.legendre.leggauss(n)
    return _t(0.5 * (a + b) + 0.5 * (b - a) * x), _t(0.5 * (b - a) * w)


def _cell(xs, x):
    """Cell index and fraction of clamped x on the ascending axis xs (both may
    carry matching batch dimensions)."""
    n = xs.shape[-1]
    if xs.dim() == 1:
        x = x.clamp(min=float(xs[0]), max=float(xs[-1]))
        i = (torch.searchsorted(xs, x.contiguous(), right=True) - 1).clamp(0, n - 2)
        return i, (x - xs[i]) / (xs[i + 1] - xs[i])
    x = torch.minimum(torch.maximum(x, xs[..., :1]), xs[..., -1:])
    i = (torch.searchsorted(xs.contiguous(), x.contiguous(), right=True) - 1).clamp(0, n - 2)
    a = torch.gather(xs, -1, i)
    return i, (x - a) / (torch.gather(xs, -1, i + 1) - a)


def _lin(xs, ys, x):
    """Clamped linear interpolation: ys [..., n], x [m] or [..., m]."""
    i, f = _cell(xs, x)
    if ys.dim() == 1:
        return ys[i] + f * (ys[i + 1] - ys[i])
    if ys.dim() > i.dim():
        i, f = i.expand(*ys.shape[:-1], -1), f.expand(*ys.shape[:-1], -1)
    a = torch.gather(ys, -1, i)
    return a + f * (torch.gather(ys, -1, i + 1) - a)


def _bilin(xs, ys, zs, x, y):
    """Clamped bilinear zs [..., ny, nx] at the outer product of y and x:
    [..., len(y), len(x)]; xs [nx] or [..., nx], ys [ny]."""
    i, t = _cell(xs, x.expand(*xs.shape[:-1], -1) if xs.dim() > 1 else x)
    j, u = _cell(ys, y)
    u = u[:, None]
    if xs.dim() > 1:
        i = i[..., None, :].expand(*zs.shape[:-2], len(y), -1)
        t = t[..., None, :]
        r0, r1 = zs[..., j, :], zs[..., j + 1, :]
        g = torch.gather
        return (1 - t) * (1 - u) * g(r0, -1, i) + t * (1 - u) * g(r0, -1, i + 1) + \
            (1 - t) * u * g(r1, -1, i) + t * u * g(r1, -1, i + 1)
    r0, r1 = zs[..., j, :], zs[..., j + 1, :]
    return (1 - t) * (1 - u) * r0[..., i] + t * (1 - u) * r0[..., i + 1] + \
        (1 - t) * u * r1[..., i] + t * u * r1[..., i + 1]


def _omega_z(z):
    def poly(c, x):
        out = torch.zeros_like(x)
        for v in c:
            out = v + x * out
        return out

    f1 = poly((-0.00262353, 0.01940118, 0.45133063), z)
    f2 = poly((1.33647377e4, 1.35291046e3, -1.26204891e2, -2.83454918e1, -2.26465905,
               3.84958753e-1), z - 0.6)
    f3 = poly((-1.88101967, 4.8071839, -4.11424324, 1.18196785), z)
    return torch.where(z < 0.504, f1, torch.where(z < 0.7, f2, f3))


def _dv(z, da, om):
    """dV/dOmega/dz of a flat universe from d_a at z (om broadcast)."""
    return 2997.92 * (1 + z) ** 2 * (da * H0) ** 2 / torch.sqrt(om * (1 + z) ** 3 + (1 - om))


def _emg_tail(x, mu, sg, tau):
    z = (x - mu) / sg
    u = (tau * sg - z) / math.sqrt(2.0)
    tail = 0.5 * torch.special.erfcx(u.abs()) * torch.exp(-0.5 * z * z)
    A = (-tau * (x - mu) + 0.5 * (tau * sg) ** 2).clamp(-700.0, 700.0)
    return torch.where(u < 0, torch.exp(A) - tail, tail)


def _dsigma(x):
    """Projected NFW Sigma_bar(<x) - Sigma(x) in units of 2 r_s delta_c rho."""
    w = 1.0 - x * x
    y = w.abs().sqrt().clamp(min=1e-8)
    g = torch.where(x < 1, torch.atanh(y.clamp(max=1 - 1e-16)), torch.atan(y)) / y
    s1 = torch.sqrt(w.clamp(min=0.0))
    x2 = x * x
    near = (2.0 / s1.clamp(min=1e-8)) * (torch.log(2.0 / x) / (1 + s1)
                                         + torch.log1p(-x2 / (2 * (1 + s1))) / x2)
    # small x: artanh(y) through ln((1 + y) / x), which keeps its digits
    g = torch.where(x < 0.5, torch.log((1 + s1) / x) / s1.clamp(min=1e-8), g)
    out = torch.where(x < 0.5, near, 2.0 * (g + torch.log(0.5 * x)) / x2) - (g - 1.0) / w
    m = w.abs() < 0.1
    if bool(m.any()):
        wm, xm = w[m], x[m]
        gs, ss = torch.zeros_like(wm), torch.zeros_like(wm)
        for k in range(20, -1, -1):
            gs, ss = 1.0 / (2 * k + 1) + wm * gs, 1.0 / (2 * k + 3) + wm * ss
        out[m] = 2.0 * (gs + torch.log(0.5 * xm)) / (xm * xm) - ss
    return out


def _mis_profile(x, sk, n_theta=64, n_s=128, s_max=20.0):
    """Miscentred Delta Sigma (gamma offsets) at x [m] with x / x_mis = sk,
    the two-panel quadrature split at s = sk."""
    th, wth = _gl(0.0, math.pi, n_theta)
    if sk < s_max:
        a, wa = _gl(0.0, sk, n_s // 2)
        b, wb = _gl(sk, s_max, n_s - n_s // 2)
        s, ws = torch.cat([a, b]), torch.cat([wa, wb])
    else:
        s, ws = _gl(0.0, s_max, n_s)
    ct, r = torch.cos(th), s[:, None] / sk          # offsets in units of x
    d2 = 1.0 + r * r - 2.0 * r * ct
    k = (ws * s * torch.exp(-s) / math.pi)[:, None] * wth * (2.0 * (1.0 - r * ct) ** 2 / d2 - 1.0)
    d = torch.sqrt(d2).reshape(-1)
    out = []
    for xc in torch.split(x, max(1, (1 << 25) // d.numel())):
        out.append(_dsigma(xc[:, None] * d) @ k.reshape(-1))
    return torch.cat(out)


def _engine_exact(w, sets, idx, n_R):
    """Counts [n, 12] and shear [n, 12, n_R] by the direct nested sums."""
    n = len(idx)
    counts = torch.zeros((n, 12), dtype=F64, device=DEV)
    shear = torch.zeros((n, 12, n_R), dtype=F64, device=DEV) if n_R else None
    coef = _plob()[1][:, 0]
    R = _radii(n_R) if n_R else []
    for g, nodes in enumerate(sets):
        n_m, n_z, n_t, n_o, n_zo = nodes
        xm, wm = _gl(*LNM, n_m)
        xz, wz = _gl(*ZT, n_z)
        xl, wl = _gl(math.log(LAM_T[0]), math.log(LAM_T[1]), n_t)
        lam = torch.exp(xl)
        sg, tau = coef[5] * lam, coef[1] / lam ** coef[0]
        K = []
        for i in range(4):
            xo, wo = _gl(LAM_EDGES[i], LAM_EDGES[i + 1], n_o)
            d = (xo[:, None] - lam) / sg
            p = 0.9 * torch.exp(-0.5 * d * d) / (math.sqrt(2 * math.pi) * sg) \
                + 0.1 * tau * _emg_tail(xo[:, None], lam, sg, tau)
            K.append(wo @ p)
        U = torch.stack(K, 1) * wl[:, None]                       # [n_t, 4]
        sz, Kj = SZ0 * (1 + xz), []
        for j in range(3):
            xo, wo = _gl(ZOB_EDGES[j], ZOB_EDGES[j + 1], n_zo)
            d = (xo[:, None] - xz) / sz
            Kj.append(wo @ (torch.exp(-0.5 * d * d) / (math.sqrt(2 * math.pi) * sz)))
        Kj = torch.stack(Kj)                                       # [3, n_z]
        pts = [p for p in range(n) if idx[p] == g]
        # (lnM, z_t, lam_t) nodes with one exponential each
        for p in pts:
            om, s = float(w["om"][p]), float(w["sigma"][p])
            hmf = _bilin(torch.log(w["hmf_m_h"][p] * om), w["hmf_z"], w["dn"][p], xm, xz)
            mu = (float(w["B"][p]) * (xm - math.log(3e14))) \
                + (float(w["A"][p]) + 0.5 * torch.log1p(xz))[:, None]
            a, b = (xl.new_tensor(math.log(LAM_T[0])) - mu) / s, (math.log(LAM_T[1]) - mu) / s
            e2, ecx = math.sqrt(2.0), torch.special.erfcx
            # D exp(v^2 / 2) with v the distance to the domain (0 inside it)
            lo = 0.5 * (ecx(a.clamp(min=0) / e2)
                        - ecx(b.clamp(min=0) / e2) * torch.exp(-0.5 * (b * b - a * a).clamp(min=0)))
            up = 0.5 * (ecx((-b).clamp(min=0) / e2) - ecx((-a).clamp(min=0) / e2)
                        * torch.exp(-0.5 * (a * a - b * b).clamp(min=0)))
            D = torch.where(a > 0, lo, torch.where(b < 0, up, 1 - 0.5 * torch.erfc(-a / e2)
                                                   - 0.5 * torch.erfc(b / e2)))
            v2 = torch.where(a > 0, a * a, torch.where(b < 0, b * b, torch.zeros_like(a)))
            S = torch.exp(-0.5 * (((xl - mu[..., None]) / s) ** 2 - v2[..., None])) @ U
            V = (hmf / (math.sqrt(2 * math.pi) * s * D))[..., None] * S   # [n_z, n_m, 4]
            da = _lin(w["dist_z"], w["dist_da"][p], xz)
            c = wz * _dv(xz, da, om) * _omega_z(xz)
            W = torch.einsum("jq,qki->jik", Kj * c, V).reshape(12, n_m)
            counts[p] = W @ wm
            if n_R:
                cs = c * _lin(w["sci_z"], w["sci_val"][p], xz)
                w["_Wg", p] = torch.einsum("jq,qki->jik", Kj * cs, V).reshape(12, n_m) * wm
        if not n_R or not pts:
            continue
        om = _t(w["om"][pts])[:, None]
        conc = 5.0 * (torch.exp(xm) / 1e14) ** -0.1
        rs = ((3 * torch.exp(xm) / (800 * math.pi * RHO_CRIT * om)) ** (1.0 / 3.0)) / conc
        dc = (200 * conc ** 3 / 3) / (torch.log(1 + conc) - conc / (1 + conc))
        norm = 2 * rs * dc * RHO_CRIT * om * 1e-12
        Wg = torch.stack([w.pop(("_Wg", p)) for p in pts])          # [np, 12, n_m]
        at = torch.tensor(pts, device=DEV)
        for r in range(n_R):
            x = R[r] / rs
            cen = _dsigma(x)
            for i in range(4):
                sk = float(R[r]) / (0.17 * (LOB[i] / 100.0) ** 0.2)
                phi = norm * (0.8 * cen + 0.2 * _mis_profile(x.reshape(-1), sk).reshape(x.shape))
                for j in range(3):
                    shear[at, i + 4 * j, r] = (Wg[:, i + 4 * j] * phi).sum(1)
    return counts, shear


def _exact_engine(case, seed):
    sets = _node_sets(case)
    idx = _grid_index(case["n"], len(sets))
    w = _walkers(case["n"], seed, sci=case["radii"] > 0)
    if case["hmf_fp32"]:
        w["dn"] = w["dn"].float().double()
    counts, shear = _engine_exact(w, sets, idx, case["radii"])
    if not case["radii"]:
        return [counts]
    if not case["loglike"]:
        return [counts, shear]
    d, ic, s, ics = (_t(v) for v in _data_vector(case, seed))
    th = torch.where(counts[:, :, None] > 0, shear / counts[:, :, None], torch.zeros_like(shear))
    chi2 = ((d - counts) ** 2 * ic).sum(1) + ((s - th.flatten(1)) ** 2 * ics).sum(1)
    return [counts, shear, -0.5 * chi2]


def _exact_serve(case, seed):
    sizes = _request_sizes(case)
    n = int(sizes.sum())
    w = _walkers(n, seed, sci=False)
    w["dn"] = w["dn"].float().double()
    counts, _ = _engine_exact(w, [DENSITY[d] for d in (1, 2, 4)], np.arange(n) % 3, 0)
    return list(torch.split(counts, [int(m) for m in sizes]))


def _cdf(x):
    return 0.5 * (1 + torch.erf(x / math.sqrt(2.0)))


def _exact_module(case, seed):
    s = _module_inputs(case, seed)
    c, mor, t = s["cfg"], s["mor"], {k: _t(v) for k, v in s["tab"].items()}
    om = s["om"]
    lnM = _t(np.linspace(c["lnm_low"], c["lnm_high"], c["n_lnm"]))
    z = _t(np.linspace(c["zt_low"], c["zt_high"], c["n_z"]))
    gx, gw = _gl(-1.0, 1.0, c["n_q"])
    L, Z = lnM[:, None], z[None, :]
    M = torch.exp(L)
    if s["kind"] == 0:
        Mmin, M1 = 10.0 ** mor[0], 10.0 ** mor[1]
        base = (M - Mmin).clamp(min=0) / (M1 - Mmin)
        ms = base ** mor[2] * ((1 + Z) / (1 + mor[5])) ** mor[3]
        cen = (M >= Mmin).double() + 0 * Z
        mu, de = cen + ms, (mor[4] * ms) ** 2
        sd = torch.sqrt(ms + de)
        lo, hi = (mu - 6 * sd).clamp(min=0), mu + 6 * sd
    else:
        mu = mor[0] + mor[1] * (L - math.log(mor[4])) + mor[2] * torch.log1p(Z)
        lo = torch.exp(mu - 6 * mor[3]).clamp(min=mor[5])
        hi = torch.exp(mu + 6 * mor[3]).clamp(max=mor[6])
        D = _cdf((math.log(mor[6]) - mu) / mor[3]) - _cdf((math.log(mor[5]) - mu) / mor[3])
    half, mid = (0.5 * (hi - lo))[..., None], (0.5 * (hi + lo))[..., None]
    lt, W = mid + half * gx, half * gw
    if s["kind"] == 0:
        msx, dex, cx = ms[..., None], de[..., None], cen[..., None]
        x = lt - cx + dex
        P = torch.exp(-(msx + dex) + (x - 1) * torch.log((msx + dex).clamp(min=1e-300))
                      - torch.lgamma(x.clamp(min=1e-300)))
        P = torch.where(x > 0, P, torch.zeros_like(P))
        P = torch.where(msx <= 1e-8, torch.exp(-0.5 * ((lt - cx) / 1e-3) ** 2)
                        / (math.sqrt(2 * math.pi) * 1e-3), P)
        P = torch.where((lt < 0) | (lt < cx), torch.zeros_like(P), P)
    else:
        dd = (torch.log(lt) - mu[..., None]) / mor[3]
        P = torch.exp(-0.5 * dd * dd) / (math.sqrt(2 * math.pi) * mor[3] * lt * D[..., None])
    pz, pc = _t(s["plob"][0]), _t(s["plob"][1])
    a_tau, b_tau, a_mu, b_mu, a_sg, b_sg, a_f, b_f = \
        (v[None, :, None] for v in _lin(pz, pc, z))
    pm, psg, ptau = a_mu + b_mu * lt, b_sg * lt ** a_sg, b_tau / lt ** a_tau
    pf = (b_f / (1 + torch.exp(-lt)) ** a_f).clamp(max=1.0)
    cdf = [(_cdf((e - pm) / psg) - pf * _emg_tail(torch.full_like(pm, e), pm, psg, ptau))
           .clamp(0.0, 1.0) for e in LAM_EDGES]
    Si = [torch.where(hi > lo, (W * (cdf[i + 1] - cdf[i]) * P).sum(-1), torch.zeros_like(lo))
          for i in range(4)]
    S = []
    for k in range(12):
        kj = _cdf((c["zob_max"][k] - z) / 0.03) - _cdf((c["zob_min"][k] - z) / 0.03)
        S.append((Si[k % 4] * kj).T)
    S = torch.stack(S)                                             # [12, n_z, n_lnM]
    xm, wm = _gl(29.9336, 36.73, case["n_lnm"])
    xz, wz = _gl(0.05, 0.8, case["n_z"])
    hmf = _bilin(torch.log(t["hmf_m_h"] * om), t["hmf_z"], t["dndlnmh"], xm, xz)
    zf = wz * _dv(xz, _lin(t["dist_z"], t["dist_da"], xz), om) * _omega_z(xz)
    sel = _bilin(lnM, z, S, xm, xz)                                # [12, nq, nm]
    counts = torch.einsum("q,qk,bqk->bk", zf, hmf, sel) @ wm
    Wg = torch.einsum("q,qk,bqk->bk", zf * _lin(t["sci_z"], t["sci_val"], xz), hmf, sel) * wm
    h = {k: _t(v) for k, v in s["halo"].items()}
    R = _radii(case["radii"])
    cen = _bilin(h["r_sigma"], h["lnM"], h["dSigma_nfw"], _t(R), xm)   # [nm, nR]
    rs = (3 * torch.exp(xm) / (800 * math.pi * RHO_CRIT)) ** (1.0 / 3.0) / 4.0
    dc = (200.0 * 64.0 / 3.0) / (math.log(5.0) - 0.8)
    shear = torch.empty((12, len(R)), dtype=F64, device=DEV)
    for i in range(4):
        for r in range(len(R)):
            sk = float(R[r]) / (0.17 * (LOB[i] / 100.0) ** 0.2)
            mis = _mis_profile(R[r] / rs, sk)
            phi = 0.78 * cen[:, r] + 0.22 * (2 * rs * dc * RHO_CRIT * om * 1e-12) * mis
            for j in range(3):
                shear[i + 4 * j, r] = (Wg[i + 4 * j] * phi).sum()
    return [S, counts, shear.reshape(-1)]


# Photo-z width sigma_z(z) on 120 nodes in [0.1, 0.9].
_SZ_Z = np.round(np.linspace(0.1, 0.9, 120), 9)
_SZ = np.array([
    0.0399897614683744, 0.04045843186344669, 0.04114636168595637, 0.0420871335844959,
    0.04333171959264844, 0.04478443335373124, 0.045529454632531614, 0.04525452972432995,
    0.04410570407088478, 0.0428796455633828, 0.04211877697349987, 0.042074357794901464,
    0.042672902992802304, 0.04362443187095412, 0.044686243927015194, 0.045698673172211025,
    0.046759409894746445, 0.047979697512620725, 0.049451541881770936, 0.05111162500814543,
    0.052862309265093506, 0.05450906951472781, 0.05596050477868047, 0.05719427217767708,
    0.058333561507125806, 0.05950093818680306, 0.060748321464353196, 0.06203684049398442,
    0.06341575638352769, 0.06497966869173018, 0.06692054901053487, 0.06920866466097016,
    0.0717731947767403, 0.07440707962391233, 0.07688046965455221, 0.07898096996570447,
    0.08050805933118069, 0.08159894976555493, 0.08239243770649567, 0.08308520436442364,
    0.08379643229091648, 0.08460100672214806, 0.08556900268992938, 0.0866943385735301,
    0.08794228585742969, 0.08923580236362819, 0.09043806304910247, 0.09145268914045644,
    0.09219898293814413, 0.0927417660905204, 0.09313337444231765, 0.09341932066628694,
    0.09353072998840134, 0.09342562142811889, 0.09307289195166428, 0.09247121854851657,
    0.09164426488618577, 0.09064644539430342, 0.08964704132260966, 0.08879213966250611,
    0.08820842470461246, 0.08798057371694759, 0.08814081913479109, 0.08870041314615683,
    0.08958066774781187, 0.0906519091556056, 0.09180708080120513, 0.09306022190478362,
    0.09447838393048853, 0.09610356354010792, 0.09784603819553066, 0.09961753790169015,
    0.1013707861998071, 0.1031846682571597, 0.10511256806117333, 0.10717469971718516,
    0.10930651098717054, 0.11144532793125458, 0.11356947889755749, 0.11575529356173295,
    0.1180998897716627, 0.12066139617148375, 0.12342487619269804, 0.1263207303582879,
    0.1292665701656416, 0.1321247140940486, 0.13489263210140817, 0.13758220179317884,
    0.14023009483951568, 0.14272204160007199, 0.14494513758587016, 0.14676336450583208,
    0.14797743041022654, 0.14845169156641555, 0.1481073739698509, 0.1471711875761524,
    0.1457596650078168, 0.14391004252859188, 0.14137473952350366, 0.1382413486047733,
    0.13479868691362765, 0.13161144466485766, 0.12890315740407576, 0.12678955919979562,
    0.1250975088012601, 0.12353341316973442, 0.12170093899419578, 0.11920033791022243,
    0.11587710443589729, 0.11175743529941101, 0.1074793101300091, 0.10377908395966623,
    0.10123986697084572, 0.09977484620272835, 0.09928085950286167, 0.09971523400996213,
    0.101115431416433, 0.10360843593962064, 0.10744520713658108, 0.11308048661154518,
])


def _sigma_z(z):
    return _lin(_t(_SZ_Z), _t(_SZ), z)


def _chi_of(dz, dc):
    return lambda z: _lin(dz, dc, z) * H0


def _invert(chi, target, lo=0.001, hi=2.0):
    lo, hi = torch.full_like(target, lo), torch.full_like(target, hi)
    for _ in range(40):
        mid = 0.5 * (lo + hi)
        below = chi(mid) < target
        lo, hi = torch.where(below, mid, lo), torch.where(below, hi, mid)
    return 0.5 * (lo + hi)


def _wing(chi, chi_o, R_excl, far, sign, n):
    """Log-spaced line-of-sight nodes beyond the exclusion ring, batched."""
    x, wx = _gl(-1.0, 1.0, n)
    a, b = torch.log(R_excl), torch.log(far)
    u = 0.5 * (a + b) + 0.5 * (b - a) * x
    dis = torch.exp(u)
    z = _invert(chi, chi_o + sign * dis)
    slope = (chi(z + 1e-3) - chi(z - 1e-3)) / 2e-3
    return z, 0.5 * (b - a) * wx * dis / slope


def _los_grid(chi, zob, z_fg, z_bg, R_excl, n_ring, n_outer):
    """Front wing, ring and back wing nodes and weights [S, n]."""
    one = torch.ones_like(R_excl)
    chi_o = chi(zob * one)
    dz = R_excl / ((chi((zob + 1e-3) * one) - chi((zob - 1e-3) * one)) / 2e-3)
    lo, hi = (zob - dz).clamp(min=z_fg), (zob + dz).clamp(max=z_bg)
    x, wx = _gl(-1.0, 1.0, n_ring)
    ring, wr = 0.5 * (lo + hi) + 0.5 * (hi - lo) * x, 0.5 * (hi - lo) * wx
    zf, wf = _wing(chi, chi_o, R_excl, chi_o - chi(z_fg * one), -1.0, n_outer)
    zb, wb = _wing(chi, chi_o, R_excl, chi(z_bg * one) - chi_o, 1.0, n_outer)
    return torch.cat([zf, ring, zb], -1), torch.cat([wf, wr, wb], -1)


def _exact_prj(case, seed):
    om, t, p, grid = _prj_inputs(case, seed)
    t, p = ({k: _t(v) for k, v in d.items()} for d in (t, p))
    n_lnm, nR = case["n_lnm"], case["radii"]
    R = grid["radii"][:nR]
    lnx, lnw = _gl(*LNM, n_lnm)
    rs = (3 * torch.exp(lnx) / (800 * math.pi * RHO_CRIT)) ** (1.0 / 3.0) / 4.0
    dc = (200.0 * 64.0 / 3.0) / (math.log(5.0) - 0.8)
    norm = 2 * rs * dc * RHO_CRIT * om * 1e-12
    cth, wth = _gl(0.0, math.pi, 256)
    cth = torch.cos(cth)
    chi = _chi_of(t["dist_z"], p["dist_dc"])
    ax = torch.log(t["hmf_m_h"] * om)

    def nb(z):
        return _bilin(ax, t["hmf_z"], t["dndlnmh"], lnx, z), \
            _bilin(p["halo_lnM"], p["halo_z"], p["bias"], lnx, z)

    out = []
    for zi in range(3):
        zob = 0.5 * (ZOB_EDGES[zi] + ZOB_EDGES[zi + 1])
        chi_o = chi(_t([zob]))
        DA = float(chi_o) / (1 + zob)
        sci = float(_lin(t["sci_z"], t["sci_val"], _t([zob])))
        for lb in range(4):
            Rl = (LOB[lb] / 100.0) ** 0.2
            R_ex = Rl * (1 + zob)
            th_lam = Rl * (1 + zob) / float(chi_o)
            th_ex, th_R = R_ex / float(chi_o), R / DA
            th_max = max(30.0 / DA, 3.0 * th_R.max())
            lower = max(1e-8, 0.1 * min(th_ex, th_R.min(), th_lam))
            b = sorted(x for x in [lower, th_ex, *th_R, th_lam, 2 * th_lam, th_max] if x <= th_max)
            bp = [b[0]]
            for x in b[1:]:
                if x > bp[-1] * (1 + 1e-6):
                    bp.append(x)
            th, wt = [], []
            for x0, x1 in zip(bp[:-1], bp[1:]):
                u, wu = _gl(math.log(x0), math.log(x1), case["n_per_seg"])
                th.append(torch.exp(u))
                wt.append(wu * th[-1])
            th, wt = torch.cat(th), torch.cat(wt)
            geom = wt * 2 * math.pi * torch.sin(th)
            bs, bl = (float(p[k].reshape(3, 4)[zi, lb]) for k in ("b_small", "b_large"))
            bsel = bs + (bl - bs) / (1 + torch.exp(-2.5 / th_lam * (th - 0.5 * th_lam)))
            z, wz = _los_grid(chi, zob, 0.1, 0.8, _t([R_ex]), case["n_zring"], case["n_zouter"])
            u = (z - zob) / _sigma_z(z)
            cz = _dv(z, _lin(t["dist_z"], t["dist_da"], z), om) * _omega_z(z) * wz \
                * torch.where(u.abs() < 1, 1 - u * u, torch.zeros_like(u))
            n, bi = nb(z)
            no, bo = nb(_t([zob]))
            an = lnw * rs
            ab = cz * ((an * n * bi).sum(1) / ((an * no * bo).sum() + 1e-300))
            wrnd = (cz[:, None] * n * lnw).sum(0)
            wcl = lnw * (no * bo)[0]
            ch = chi(z)
            ce = (ch * ch + chi_o * chi_o - R_ex * R_ex) / (2 * ch * chi_o + 1e-30)
            tex = torch.where(ce >= 1 - 1e-12, torch.zeros_like(ce),
                              torch.acos(ce.clamp(-1.0, 1.0)))
            dchi = torch.sqrt((ch * ch + chi_o * chi_o
                               - 2 * ch * chi_o * torch.cos(th)[:, None]).clamp(min=0))
            xi0 = _bilin(p["xi_r"], p["xi_z"], p["xi_nl"], dchi.reshape(-1), _t([zob]))[0]
            psi = (ab * xi0.reshape(dchi.shape) * (th[:, None] > tex)).sum(1)
            xm = (th * DA)[:, None] / rs
            for r in R:
                x = float(r) / rs
                x, m = x[None, :, None], xm[..., None]
                d2 = x * x + m * m - 2 * x * m * cth
                a = x - m * cth
                v = norm * ((_dsigma(torch.sqrt(d2)) * (2 * a * a / d2 - 1)) @ wth) / math.pi
                rnd = float((geom * (v @ wrnd)).sum())
                cl = float((geom * bsel * psi * (v @ wcl)).sum())
                tot = rnd + cl
                out.append([tot, rnd, cl] + 2 * [tot * sci, rnd * sci, cl * sci])
    return np.array(out)


def _overlap(th, lo, ll):
    """Two-disk overlap fraction of radii lo and ll at distance th."""
    A = (th * th + ll * ll - lo * lo) / (2 * th * ll)
    B = (th * th + lo * lo - ll * ll) / (2 * th * lo)
    sq = (-th + ll + lo) * (th + ll - lo) * (th - ll + lo) * (th + ll + lo)
    f = (ll * ll * torch.acos(A.clamp(-1, 1)) + lo * lo * torch.acos(B.clamp(-1, 1))
         - 0.5 * torch.sqrt(sq.clamp(min=0))) / (math.pi * ll * ll)
    inside = torch.where(ll <= lo, torch.ones_like(f), (lo / ll) ** 2 + 0 * f)
    f = torch.where(th <= (lo - ll).abs(), inside, f)
    return torch.where(th > lo + ll, torch.zeros_like(f), f)


def _photoz_edge(zob, sign, lo, hi):
    for _ in range(50):
        mid = 0.5 * (lo + hi)
        if mid + sign * float(_sigma_z(_t([mid]))) < zob:
            lo = mid
        else:
            hi = mid
    return 0.5 * (lo + hi)


def _exact_bsel(case, seed):
    w, hal, hod = _bsel_inputs(case, seed)
    n, NT = case["n"], case["n_theta"]
    om, hod = _t(w["om"])[:, None], _t(hod)
    lnx, lnw = _gl(*LNM, case["n_lnm"])
    zr = _t(np.linspace(0.05, 0.90, case["n_zt_ref"]))
    chi = _chi_of(w["dist_z"], w["dist_dc"])
    hm = _bilin(torch.log(w["hmf_m_h"] * om), w["hmf_z"], w["dn"], lnx, zr)     # [n, nz, nM]
    hb = _bilin(hal["halo_lnM"], hal["halo_z"], hal["bias"], lnx, zr)
    cr, sr = chi(zr), _sigma_z(zr)
    dr = _dv(zr, _lin(w["dist_z"], w["dist_da"], zr), om)
    Mmin, M1 = 10.0 ** hod[:, :1], 10.0 ** hod[:, 1:2]
    base = ((torch.exp(lnx) - Mmin).clamp(min=0) / (M1 - Mmin)) ** hod[:, 2:3]
    zf = ((1 + zr) / 1.45) ** hod[:, 3:4]
    ls = zf[:, :, None] * base[:, None, :]
    mi = (ls * hod[:, 4, None, None]) ** 2
    lam = (ls + mi).clamp(min=1e-300)
    out = torch.empty((n, 12, 3), dtype=F64, device=DEV)
    for lb in range(4):
        lt, ltw = _gl(1e-6, LOB[lb], case["n_lt"])
        x = lt + mi[..., None]
        mor = torch.exp(-lam[..., None] + (x - 1) * torch.log(lam)[..., None] - torch.lgamma(x))
        Rl, rl = (LOB[lb] / 100.0) ** 0.2, (lt / 100.0) ** 0.2
        for zi in range(3):
            zob = 0.5 * (ZOB_EDGES[zi] + ZOB_EDGES[zi + 1])
            one = torch.ones((n, 1), dtype=F64, device=DEV)
            chi_o = chi(zob * one)
            R_ex = Rl * (1 + zob) * one
            th_lob = Rl * (1 + zob) / chi_o
            z, wz = _los_grid(chi, zob, _photoz_edge(zob, 1.0, 0.01, zob),
                              _photoz_edge(zob, -1.0, zob, 1.5), R_ex, case["n_zring"],
                              case["n_zouter"])
            u = (z - 0.05) / (0.85 / (case["n_zt_ref"] - 1))
            i = u.long().clamp(0, case["n_zt_ref"] - 2)
            f = u - i

            def at(v):
                v = v.expand(n, -1) if v.dim() == 1 else v
                a = torch.gather(v, 1, i)
                return a + f * (torch.gather(v, 1, i + 1) - a)

            rows = torch.arange(n, device=DEV)[:, None]

            def at2(v):
                g = f[(...,) + (None,) * (v.dim() - 2)]
                return v[rows, i] + g * (v[rows, i + 1] - v[rows, i])

            cz, dv, sg = at(cr), at(dr), at(sr)
            uu = (z - zob) / sg
            wv = torch.where(uu.abs() < 1, 1 - uu * uu, torch.zeros_like(uu))
            ce = (cz * cz + chi_o * chi_o - R_ex * R_ex) / (2 * cz * chi_o)
            tex = torch.where(ce >= 1 - 1e-12, torch.full_like(ce, 1e-6),
                              torch.acos(ce.clamp(-1.0, 1.0)))
            th_hi = 2 * th_lob
            th_lo = torch.minimum(tex.min(1, keepdim=True).values, th_hi)
            mid = torch.maximum(torch.minimum(th_lob, th_hi), th_lo)
            x1, w1 = _gl(-1.0, 1.0, NT // 2)
            x2, w2 = _gl(-1.0, 1.0, NT - NT // 2)
            h1, h2 = 0.5 * (mid - th_lo), 0.5 * (th_hi - mid)
            th = torch.cat([0.5 * (th_lo + mid) + h1 * x1, 0.5 * (mid + th_hi) + h2 * x2], 1)
            g = torch.cat([h1 * w1, h2 * w2], 1) * 2 * math.pi * torch.sin(th)
            sig = 1 / (1 + torch.exp(-2.5 / th_lob * (th - 0.5 * th_lob)))
            nM, bM, pm = at2(hm), at2(hb), at2(mor)
            pref = (wv * dv * wz)[..., None] * (lt * ltw)
            WP = pref * torch.einsum("szm,szml->szl", lnw * nM, pm)
            WI = pref * torch.einsum("szm,szml->szl", lnw * nM * bM, pm)
            xz = hal["xi_z"]
            q = (zob - float(xz[0])) / float(xz[1] - xz[0])
            j = min(max(int(math.floor(q)), 0), len(xz) - 2)
            xi0 = hal["xi_nl"][:, j] + (q - j) * (hal["xi_nl"][:, j + 1] - hal["xi_nl"][:, j])
            r = hal["xi_r"]
            dchi = torch.sqrt((cz * cz + chi_o * chi_o)[:, None, :]
                              - (2 * cz * chi_o)[:, None, :] * torch.cos(th)[..., None])
            v = (torch.log(dchi.clamp(min=float(r[0]), max=float(r[-1]))) - math.log(float(r[0]))) \
                / math.log(float(r[1] / r[0]))
            k = v.floor().long().clamp(0, len(r) - 2)
            flat = k.reshape(n, -1)
            a0 = torch.gather(xi0, 1, flat).reshape(k.shape)
            a1 = torch.gather(xi0, 1, flat + 1).reshape(k.shape)
            xi = a0 + (v - k) * (a1 - a0)
            fA = _overlap(th[:, :, None, None], th_lob[:, :, None, None],
                          (rl * ((1 + z) / cz)[..., None])[:, None])
            on = (th[..., None] > tex[:, None, :]).double()
            sP = ((fA * WP[:, None]).sum(-1) * on).sum(-1)
            sI = ((fA * WI[:, None]).sum(-1) * on * xi).sum(-1)
            o = lb + 4 * zi
            out[:, o, 0] = (g * sP).sum(1)
            out[:, o, 1] = (g * sig * sI).sum(1)
            out[:, o, 2] = (g * (1 - sig) * sI).sum(1)
    return out


def exact(case, seed):
    f = {"engine": _exact_engine, "serve": _exact_serve, "module": _exact_module,
         "prj": _exact_prj, "bsel": _exact_bsel}[case["kind"]]
    return f(case, seed)
