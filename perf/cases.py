"""The work that users of this package have it do, as cases to be timed.

Each case is one pass through the public entry points (``gpu.Model``,
``mlp.Mlp``) on inputs made from a seed: a run of days on a region, the
per-day calls of the reference's day loop, or the calibration network.  A pass
over the same state goes on from where the last one ended, as a spin-up over
one period does.

``exact`` computes the same outputs in 64 bits with plain torch: the day's
vertical balance (daily.cpp:94-1257, lai.cpp:152-293) and routing
(routing.cpp:1835-4520, 5034-5188) over all cells at once, cell n's day d at
step d + offset(n) so that its upstream cells' day d is there.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from watergap2_gb300 import synthetic
from watergap2_gb300.gpu import Model
from watergap2_gb300.mlp import Mlp

STATE = ("canopy", "soil", "snow", "snow_band", "lai_days", "lai_status", "lai_precsum", "gw", "river", "loclake",
         "locwetl", "glolake", "glowetl", "res", "rf_loclake", "rf_locwetl", "rf_glolake", "rf_glowetl", "rf_res",
         "k_release", "laf", "laf_prev", "fswb_next", "laf_started")
# what integrate_wghm_ reads back at a month's end (integrateWGHM.cpp:830-847)
MONTH_END = ("canopy", "soil", "snow", "snow_band", "laf")
# the monthly grids a run of the output case writes
GRIDS = ("river_avail", "storage", "cell_runoff", "prec", "temp", "pet", "aet", "swe", "soil_wc", "runoff",
         "gw_recharge", "open_water_evap")
DOY0 = 60   # the first simulated day of the year
FIRST = (1, 32, 60, 91, 121, 152, 182, 213, 244, 274, 305, 335)   # the first day of each month


def _case(name, kind, grid, size, days, per_step=1, precision="fp64", members=1, option="plain", velo=1):
    return dict(name=name, kind=kind, grid=grid, size=size, days=days, per_step=per_step, precision=precision,
                members=members, option=option, velo=velo)


def listed():
    return [
        # a test basin for a month: the smallest run, all latency
        _case("basin_month", "run", "block", 16, 30),
        # one region without water bodies for a year, as the 64 x 64 configuration
        _case("region_year", "run", "block", 64, 365),
        # the reference's own day loop on a small region with every kind of water
        # body: two calls a day, the model read at the month's end
        _case("lakes_day_loop", "day_loop", "lakes", 24, 31, velo=2),
        # the same loop on the global half-degree grid
        _case("global_day_loop", "day_loop", "global", 67420, 3),
        # the headline: the global grid for a year in one call, checkpoint at the end
        _case("global_year", "run", "global", 67420, 365, per_step=5),
        # half a year with a dozen monthly grids written
        _case("global_grids", "run", "global", 67420, 181, per_step=5, option="grids"),
        # half a year with water use met in the cells
        _case("global_use", "run", "global", 67420, 181, per_step=5, option="use"),
        # half a year with water temperature and fractional routing
        _case("global_temp", "run", "global", 67420, 181, per_step=5, option="temp"),
        # a finer grid in single precision
        _case("fine_single", "run", "global", 550000, 90, per_step=5, precision="fp32"),
        # a batch of perturbed members, discharge at the gauges
        _case("ensemble", "run", "global", 67420, 90, per_step=5, precision="fp32", members=64),
        # the calibration network: a proposal for every basin, and a gradient
        _case("network_forward", "forward", "none", 1000, 0),
        _case("network_gradient", "gradient", "none", 16384, 0),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(("block", "lakes", "day_loop", "global", "global", "option", "single", "ensemble", "network"))
    if what == "block":
        return _drawn("run", "block", rng.randint(9, 64), spread(5, 365), rng.choice((1, 1, 3, 5)))
    if what == "lakes":
        return _drawn("run", "lakes", rng.randint(13, 40), spread(5, 365), rng.choice((1, 1, 4, 5)), velo=rng.choice((1, 2)))
    if what == "day_loop":
        if rng.random() < 0.5:
            return _drawn("day_loop", "lakes", rng.randint(13, 40), rng.randint(3, 31), velo=rng.choice((1, 2)))
        return _drawn("day_loop", "global", spread(9000, 67420), rng.randint(1, 3))
    if what == "global":
        return _drawn("run", "global", spread(5000, 67420), rng.randint(20, 365), rng.randint(1, 7), velo=rng.choice((1, 1, 2)))
    if what == "option":
        return _drawn("run", "global", spread(5000, 67420), rng.randint(20, 181), rng.randint(1, 7),
                      option=rng.choice(("grids", "use", "temp")))
    if what == "single":
        return _drawn("run", "global", spread(30000, 550000), rng.randint(10, 90), rng.choice((1, 5)), precision="fp32")
    if what == "ensemble":
        members = spread(2, 64)
        return _drawn("run", "global", spread(5000, 67420), rng.randint(10, 90), rng.choice((1, 5)), precision="fp32",
                      members=members)
    return _drawn(rng.choice(("forward", "gradient")), "none", spread(100, 16384), 0)


def _drawn(kind, grid, size, days, per_step=1, **kw):
    c = _case("", kind, grid, size, days, per_step, **kw)
    del c["name"]
    return c


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=4)
def _region(grid, size, velo, frac):
    if grid == "block":
        return synthetic.region_64x64(size=size)
    if grid == "lakes":
        return synthetic.region_small_swb(ny=size, nx=2 * size, river_velo_opt=velo)
    k = size / 67420.0
    ny = max(60, int(round(360 * math.sqrt(k))))
    r = synthetic.region_global(nland=size, n_outlets=max(8, int(6000 * k)), n_sinks=max(4, int(60 * k)),
                                swb=(int(2023 * k), int(1348 * k), max(3, int(300 * k)), max(4, int(1200 * k))),
                                river_velo_opt=velo, shape=(ny, 2 * ny))
    return r.with_options(frac_routing=1) if frac else r


def _case_region(case):
    return _region(case["grid"], case["size"], case["velo"], case["option"] == "temp")


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _weather(region, days, seed):
    """Day-major float32 precipitation, temperature, shortwave with the seasons and
    noise of synthetic.forcing, drawn on the GPU."""
    g = torch.Generator(_device()).manual_seed(seed)
    n, dev = region.ncell, _device()
    lat = torch.as_tensor(region.lat_deg, device=dev)
    hemi = torch.where(lat >= 0, 1.0, -1.0)
    tmean = 10.0 + (14.0 * (1.0 - lat.abs() / 45.0) if region.name == "region_global" else 0.0 * lat)
    doy = torch.as_tensor([(DOY0 - 1 + d) % 365 + 1 for d in range(days)], device=dev, dtype=torch.float64)[:, None]
    wet = torch.rand((days, n), generator=g, device=dev) >= 0.6
    P = torch.empty((days, n), device=dev).exponential_(1.0 / 6.4, generator=g) * wet
    T = tmean + 12.0 * torch.sin(2 * math.pi * doy / 365.0) * hemi
    T = (T + 3.0 * torch.randn((days, n), generator=g, device=dev)).float()
    S = 175.0 + 125.0 * torch.sin(2 * math.pi * (doy - 80) / 365.0) * ((lat.abs() / 30.0).clamp(0.3, 1.0) * hemi)
    S = (S + 10.0 * torch.randn((days, n), generator=g, device=dev)).clamp(50.0, 300.0).float()
    return tuple(x.cpu().numpy() for x in (P, T, S))


def _members(case, seed):
    if case["members"] == 1:
        return None, None
    rng = np.random.default_rng(seed)
    pf = np.exp(rng.normal(0.0, 0.3, case["members"])).astype(np.float32)
    gf = rng.uniform(0.7, 1.3, case["members"]).astype(np.float32)
    pf[0] = gf[0] = 1.0
    return pf, gf


def _stations(case, region):
    """Every cell in the day loop, 256 gauges (the outlets of the largest basins) for
    an ensemble, else every outlet."""
    if case["kind"] == "day_loop":
        return np.arange(region.ncell, dtype=np.int32)
    outlets = np.nonzero(region.downstream < 0)[0].astype(np.int32)
    if case["members"] == 1:
        return outlets
    cells = np.ones(region.ncell, np.int64)
    for i in region.rout_order:
        if region.downstream[i] >= 0:
            cells[region.downstream[i]] += cells[i]
    return np.sort(outlets[np.argsort(-cells[outlets], kind="stable")[:256]])


def _months(days):
    """The month of each simulated day, counted from the first one's."""
    month = [12 * (d // 365) + sum(d % 365 + 1 >= f for f in FIRST) for d in range(DOY0 - 1, DOY0 - 1 + days)]
    return [m - month[0] for m in month]


def _network(case, seed):
    """Features of basins (eleven used, the rest zero), targets and parameters (He-uniform)."""
    rng = np.random.default_rng(seed)
    x = np.zeros((case["size"], 128), np.float32)
    x[:, :11] = rng.normal(0.0, 1.0, (case["size"], 11))
    target = rng.normal(0.0, 0.5, (case["size"], 2)).astype(np.float32)
    parts = []
    for out in (128, 128, 128, 16):
        b = math.sqrt(6.0 / 128)
        parts += [rng.uniform(-b, b, out * 128), rng.uniform(-0.05, 0.05, out)]
    return x, target, np.concatenate(parts).astype(np.float32)


def prepare(case, seed):
    if case["grid"] == "none":
        x, target, theta = _network(case, seed)
        net = Mlp(seed=1)
        net.set_params(theta)
        return dict(case=case, net=net, x=x, target=target)
    region = _case_region(case)
    days, option = case["days"], case["option"]
    P, T, S = _weather(region, days, seed)
    stations = _stations(case, region)
    pf, gf = _members(case, seed)
    m = Model(region, max_days=days, stations=stations, precision=case["precision"], members=case["members"],
              prec_factor=pf, gamma_factor=gf, days_per_step=case["per_step"], water_temp=option == "temp",
              water_use=option == "use", block_threads=128 if case["members"] > 1 else 0)
    m.upload_forcing(0, P, T, S)
    if option == "use":
        years = (DOY0 - 1 + days - 1) // 365 + 1
        *use, share = synthetic.water_use_inputs(region, years, seed=seed)
        m.set_water_use_inputs(share)
        m.upload_water_use_run(0, DOY0, days, use)
    elif option == "temp":
        lw, ground = synthetic.water_temp_inputs(region, days, T, seed=seed)
        m.upload_longwave(0, lw)
        m.set_water_temp_inputs(ground)
    elif option == "grids":
        m.monthly_outputs(_months(days)[-1] + 1, doy_day0=DOY0)
        m.monthly_outputs_vertical(True)
        m.monthly_outputs_routing(True)
    m.synchronize()
    pinned = torch.empty((days, stations.size, case["members"]), dtype=torch.float64, pin_memory=True)
    return dict(case=case, model=m, discharge=pinned.numpy())


# ---------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    if case["kind"] == "forward":
        return {"y": state["net"].forward(state["x"])}
    if case["kind"] == "gradient":
        grad, loss = state["net"].gradient(state["x"], state["target"])
        return {"gradient": grad, "loss": np.float32(loss)}
    m, days = state["model"], case["days"]
    if case["kind"] == "day_loop":
        for d in range(days):
            doy = (DOY0 - 1 + d) % 365 + 1
            m.step_vertical(doy, d)
            m.step_routing(doy, d)
        out = {"state": m.get_state(fields=MONTH_END)}
    else:
        m.run_days(DOY0, 0, days)
        out = {}
        if case["option"] == "grids":
            out["grids"] = {k: m.monthly(k) for k in GRIDS}
        elif case["option"] == "use":
            out["use"] = m.water_use()
        elif case["option"] == "temp":
            out["temp"] = m.water_temp()
        if case["members"] == 1:
            out["state"] = m.get_state()
    out["discharge"] = m.discharge_into(0, days, state["discharge"])
    if case["precision"] == "fp32":   # kept in the precision that it was computed in
        out["discharge"] = out["discharge"].astype(np.float32)
        for k, a in out.get("state", {}).items():
            if a.dtype == np.float64:
                out["state"][k] = a.astype(np.float32)
    return out


def work(case):
    """Each input read once and each output written once; the operations of one
    cell-day as the reference's expressions count them (an exp or pow about 20)."""
    n, days, members = case["size"], case["days"], case["members"]
    if case["grid"] == "none":
        flops = 2.0 * n * (3 * 128 * 128 + 16 * 128)
        if case["kind"] == "forward":
            return {"bytes": 4.0 * (n * 128 + n * 16 + 51728), "flops": flops}
        return {"bytes": 4.0 * (n * 128 + n * 2 + 2 * 51728), "flops": 3.0 * flops}
    cells = {"block": n * n, "lakes": int(1.1 * n * n), "global": n}[case["grid"]]
    word = 8 if case["precision"] == "fp64" else 4
    outlets = cells if case["kind"] == "day_loop" else (256 if members > 1 else max(1, cells // 11))
    b = 12.0 * cells * days + 8.0 * outlets * days * members + 2.0 * word * 29 * cells * members
    f = 390.0
    if case["option"] == "temp":
        b, f = b + 4.0 * cells * days + 192.0 * cells, f + 200.0
    elif case["option"] == "use":
        b, f = b + 2 * 104.0 * cells, f + 15.0
    elif case["option"] == "grids":
        b, f = b + 8.0 * len(GRIDS) * cells * (_months(days)[-1] + 1), f + 40.0
    return {"bytes": b, "flops": f * cells * days * members}


# ---------------------------------------------------------------- 64 bits
def exact(case, seed):
    if case["grid"] == "none":
        return _exact_network(case, seed)
    region = _case_region(case)
    if case["option"] == "use" or region.ncell * case["members"] > 6_000_000:
        return None   # water use is not restated here
    q, state, grids = _simulate(region, _weather(region, case["days"], seed), case, seed)
    if case["kind"] == "day_loop":
        return {"state": {k: state[k] for k in MONTH_END}, "discharge": q}
    out = {"discharge": q}
    if case["members"] == 1:
        out["state"] = state
    if case["option"] == "grids":
        out["grids"] = grids
    elif case["option"] == "temp":
        out["temp"] = None   # nor the water temperature: discharge and storages are as without it
    return out


def _exact_network(case, seed):
    x, target, theta = (torch.as_tensor(a, device=_device(), dtype=torch.float64) for a in _network(case, seed))
    theta.requires_grad_(case["kind"] == "gradient")
    h, at = x, 0
    for k, out in enumerate((128, 128, 128, 16)):
        w, b = theta[at:at + out * 128].view(out, 128), theta[at + out * 128:at + out * 129]
        at += out * 129
        h = h @ w.T + b
        if k < 3:
            h = torch.relu(h)
    if case["kind"] == "forward":
        return {"y": h.cpu().numpy()}
    loss = (h[:, :2] - target).square().sum() / case["size"]
    loss.backward()
    return {"gradient": theta.grad.cpu().numpy(), "loss": float(loss)}


def _ext_rad(day, lat_deg):
    """calc_ext_rad (daily.cpp:2398-2449); day: the day of the year of each cell."""
    dec = torch.asin(0.39795 * torch.cos(0.2163108 + 2. * torch.atan(0.9671396 * torch.tan(0.00860 * (day - 186.)))))
    theta = lat_deg * (math.pi / 180.0)
    up, across = torch.sin(theta) * torch.sin(dec), torch.cos(theta) * torch.cos(dec)
    w = math.pi - torch.acos((up / across).clamp(-1.0, 1.0))
    return 15.392 * (1. + 0.033 * torch.cos(2. * math.pi / 365.0 * day)) * (w * up + across * torch.sin(w))


class _Cells:
    """Per-cell constants and state of a region, cells sorted by wavefront offset,
    [cells, 1] and [cells, members] float64; cut(lo, hi) is the same for some cells."""

    def __init__(self, values=None):
        self.__dict__.update(values or {})

    def cut(self, lo, hi):
        return _Cells({k: v[:, lo:hi] if k in ("band", "band_el") else v[lo:hi] if torch.is_tensor(v) else v
                       for k, v in self.__dict__.items()})


def _offsets(region):
    depth = np.zeros(region.ncell, np.int64)
    for i in region.rout_order[::-1]:
        if region.downstream[i] >= 0:
            depth[i] = depth[region.downstream[i]] + 1
    return depth.max() - depth


def _constants(r, order, dev, members, gf):
    n, lct = r.ncell, r.lct.astype(int) - 1

    def col(a):
        return torch.as_tensor(np.ascontiguousarray(np.asarray(a, np.float64)[order]), device=dev)[:, None]

    def flag(a):
        return torch.as_tensor(np.ascontiguousarray(np.asarray(a, bool)[order]), device=dev)[:, None]

    c = _Cells(dict(members=members, nband=r.nband, velo=r.river_velo_opt, default_velocity=r.default_velocity,
                    frac=int(r.frac_routing)))
    p = r.param
    arid = r.aindex == 1
    lake_d, wet_d = p("P_LAK_D") * 0.001, p("P_WET_D") * 0.001
    lmin = (r.lct_lai_a[lct] + r.lct_lai_b[lct] * r.lai_max).astype(np.float32)
    cont = np.maximum(r.contfreq, r.loc_lake + r.glo_lake + r.glo_res)
    bankfull = np.maximum(r.bankfull, 0.05)
    bw = 2.71 * bankfull ** 0.557 - 4.0 * (0.349 * bankfull ** 0.341)
    has_res = r.res_area > 0.
    with np.errstate(all="ignore"):
        ratio = r.stor_cap / (r.mean_outflow * 31536000. / 1e9)
    release = np.where(r.res_type == 1, np.where(r.mean_demand >= 0.5 * r.mean_outflow, 0.5 * r.mean_outflow,
                                                 r.mean_outflow - r.mean_demand), r.mean_outflow)
    for k, v in dict(lat=r.lat_deg, area=r.area_km2, cont=cont, cfa=p("P_CFA"), mprec=p("M_PREC"),
                     alpha=np.where(arid, p("P_PTC_ARI"), p("P_PTC_HUM")), max_pet=p("P_PET_MXDY"), netrad=p("M_NETRAD"),
                     mcwh=p("P_MCWH"), snowfz=p("P_T_SNOWFZ"), snowmt=p("P_T_SNOWMT"), pcrit=p("P_PCRITGWA"),
                     gamma=p("P_GAMRUN_C"), albedo=r.lct_albedo[lct], albedo_snow=r.lct_albedo_snow[lct],
                     ddf=p("M_DEGDAY_F") * r.lct_ddf[lct], lai_min=lmin, lai_max=r.lai_max, smax=r.smax, fg=r.gw_factor,
                     rgmax=r.rg_max / 100., built=r.built_up, gradnt=p("P_T_GRADNT"), kg=p("P_GWOUTF_C"), ks=p("P_SWOUTF_C"),
                     evx=p("M_EVAREDEX") * 3.32193, init=r.lct_initial_days[lct], ll=r.loc_lake / 100., lw=r.loc_wetl / 100.,
                     gw_pct=r.glo_wetl / 100., la6=r.lake_area / 1e6, ra6=r.res_area / 1e6,
                     max_ll=r.loc_lake / 100. * r.area_km2 * lake_d, max_lw=r.loc_wetl / 100. * r.area_km2 * wet_d,
                     max_gl=r.lake_area * lake_d, max_gw=r.glo_wetl / 100. * r.area_km2 * wet_d, max_res=r.stor_cap,
                     c_ratio=np.where(has_res, ratio, 1.), release=release, start=r.start_month, bw=bw,
                     mr=1. / (p("M_RIVRGH_C") * r.roughness), slope=np.sqrt(r.river_slope), length=r.river_length,
                     fcatch=np.minimum(1., (r.loc_lake + r.loc_wetl + r.glo_wetl) / 100. * 20.)).items():
        setattr(c, k, col(v))
    if gf is not None:
        c.gamma = c.gamma * torch.as_tensor(gf, device=dev, dtype=torch.float64)[None, :]
    for k, v in dict(arid=arid, arid_gw=arid & (r.texture < 21), sink=r.ldd < 0, evergreen=r.lct <= 2,
                     has_ll=r.loc_lake > 0, has_lw=r.loc_wetl > 0, has_gl=r.lake_area > 0, has_res=has_res,
                     has_gw=r.glo_wetl > 0).items():
        setattr(c, k, flag(v))
    el = r.elev.reshape(n, r.nband + 1).astype(np.float64)[order]
    c.elev0 = torch.as_tensor(el[:, :1].copy(), device=dev)
    c.band_el = torch.as_tensor(np.ascontiguousarray(el[:, 1:].T)[:, :, None], device=dev)
    # start of the run (routing.cpp:5651-5737, 807-812; annualInit)
    one = torch.ones((n, members), device=dev, dtype=torch.float64)
    laf = np.maximum(0., cont - (r.glo_lake + r.glo_wetl + r.loc_lake + r.loc_wetl + r.glo_res))
    for k in ("canopy", "soil", "snow", "lai_precsum", "gw", "rf_res", "laf_prev", "lai_days", "lai_status", "started"):
        setattr(c, k, 0. * one)
    c.band = torch.zeros((r.nband, n, members), device=dev, dtype=torch.float64)
    c.loclake, c.locwetl, c.glolake, c.glowetl = c.max_ll * one, c.max_lw * one, c.max_gl * one, c.max_gw * one
    c.res = torch.where(c.has_res, c.max_res, 0. * c.max_res) * one
    for k in ("rf_loclake", "rf_locwetl", "rf_glolake", "rf_glowetl"):
        setattr(c, k, 1. * one)
    c.k_release = 0.1 * one
    c.laf, c.fswb = col(laf) * one, (c.ll + c.lw + c.gw_pct) * one
    wbf, dbf = 2.71 * bankfull ** 0.557, 0.349 * bankfull ** 0.341
    river = r.river_length * 0.5 * dbf / 1000. * (bw / 1000. + wbf / 1000.) if r.river_velo_opt == 2 else 0. * wbf
    c.river = col(river) * one
    return c


def _tiny(x):
    return torch.where(x.abs() <= 1e-15, 0. * x, x)


def _lai(c, T, prec):
    """getDailyLai (lai.cpp:152-293)."""
    days, status, psum, init = c.lai_days, c.lai_status, c.lai_precsum, c.init
    warm, off = T > 8.0, status == 0
    rise = off & torch.where(warm, days >= init, days > init)
    wait = off & ~rise
    fall = ~off & (days <= 30)
    peak = ~off & ~fall
    dry = c.arid & (prec < 0.5)
    psum.add_(torch.where(off, prec, 0. * prec))
    d1 = days + 1.
    full = rise & (psum > 40.)
    done = full & (d1 >= init + 30.)
    d_rise = torch.where(done, init + 30., torch.where(full, d1, init + 0. * d1))
    d_fall = days - 1.
    end = fall & (d_fall <= 0.)
    d_fall = torch.where(end, 0. * d_fall, d_fall)
    d_peak = torch.where(warm & ~dry, 30. + init, days - 1.)
    new = torch.where(rise, d_rise, torch.where(wait, torch.where(warm, d1, days), torch.where(fall, d_fall, d_peak)))
    span = c.lai_max - c.lai_min
    lai = torch.where(full, c.lai_min + span * (new - init) / 30., c.lai_min + 0. * new)
    lai = torch.where(fall, c.lai_max - span * (30. - new) / 30., lai)
    lai = torch.where(peak, c.lai_max + 0. * lai, lai)
    status.copy_(torch.where(done, 1. + 0. * status, torch.where(end | (fall & warm & c.evergreen), 0. * status, status)))
    psum.copy_(torch.where(end, 0. * psum, psum))
    days.copy_(new)
    return lai


def _vertical(c, P, T, S, day):
    """calcNewDay (daily.cpp:94-1257): surface runoff, recharge, transfer, open-water
    precipitation and PET, and the terms of the monthly grids."""
    where, zero = torch.where, torch.zeros_like(c.canopy)
    laf = c.laf
    prev = where(c.started == 1, c.laf_prev, laf)
    land = laf > 0
    prec = c.mprec * P + zero
    es = 0.6108 * torch.exp(17.27 * T / (T + 237.3))
    lai = _lai(c, T, prec)
    albedo = where(c.snow > 3., c.albedo_snow, c.albedo)
    heat = where(T > 0, 2.501 - 0.002361 * T, 2.835 + 0. * T)
    solar = 0.0864 / heat * S
    ext = _ext_rad(day, c.lat)
    frac = where(ext == 0, 0. * solar, (solar / (0.75 * ext)).clamp(max=1.))
    ff = where(c.arid, 1.35 * frac - 0.35, frac)
    net_lw = -ff * (-0.02 + 0.261 * torch.exp(-0.000777 * T * T)) * 4.903e-9 * (T + 273.2) ** 4 / heat
    net = c.netrad * (solar * (1. - albedo) + net_lw)
    open_net = solar * (1. - 0.08) + net_lw
    svp = 4098. * es / (T + 237.3) ** 2
    apet = c.alpha * (svp / (svp + 0.0016286 * 101.3 / heat))
    pet = (apet * net).clamp(min=0.) + zero
    open_pet = (apet * open_net).clamp(min=0.) + zero
    ratio = where(land, prev / where(land, laf, 1. + zero), zero)
    # interception (daily.cpp:825-895)
    canopy = _tiny(c.canopy * ratio)
    transfer = where(land, zero, c.canopy)
    before, leaf = canopy, lai > 0.00001
    cap = c.mcwh * lai
    gap = cap - canopy
    fits = prec < gap
    full = where(leaf, where(fits, canopy + prec, cap), canopy)
    to_soil = where(leaf, where(fits, zero, prec - gap), prec)
    evap = where(leaf, pet * (full / where(leaf, cap, 1. + zero)).clamp(min=0.) ** 0.66666666, zero)
    out = leaf & (evap > full)
    evap = where(out, full, evap)
    soil_pet = (pet - evap).clamp(min=0.)
    canopy = where(out, zero, full - evap)
    change = canopy - before
    # snow in elevation bands (daily.cpp:897-1062)
    inv = 1.0 / c.nband
    eff, snow_evap, snow_change, snow, thresh = zero, zero, zero, zero, zero
    for e in range(c.nband):
        old = c.band[e]
        sb = _tiny(old * ratio)
        first = sb
        t = T - (c.band_el[e] - c.elev0) * c.gradnt + zero
        deep = sb > 1000.
        t = where(deep & (thresh > 0), T - (thresh - c.elev0) * c.gradnt, t)
        thresh = where(deep & (thresh == 0), c.band_el[e] + zero, thresh)
        falls = t <= c.snowfz
        sb = where(falls, sb + to_soil, sb)
        gone = where(falls, torch.minimum(sb, soil_pet), zero)
        snow_evap, sb = snow_evap + gone, where(sb > soil_pet, sb - gone, where(falls, zero, sb))
        melt = where((t > c.snowmt) & (sb >= 0), torch.minimum(c.ddf * (t - c.snowmt), sb), zero)
        sb = sb - melt
        snow_change, snow = snow_change + sb - first, snow + sb
        eff = eff + where(falls, zero, to_soil) + melt
        if e == 0:
            thawed = ~falls
        transfer = transfer + where(land, zero, old * inv)
        c.band[e].copy_(where(land, sb, zero))
    snow, eff, snow_evap = snow * inv, eff * inv, snow_evap * inv
    change = change + snow_change * inv
    c.snow.copy_(where(land, snow, zero))
    # soil, runoff, recharge (daily.cpp:1068-1257)
    immediate = where(c.built > 0, 0.5 * eff * c.built, zero)
    eff = eff - immediate
    transfer = where(land, zero, (transfer + c.soil) * c.cfa)
    soil = c.soil * ratio
    before = soil
    over = (soil - c.smax).clamp(min=0.)
    soil = torch.minimum(soil, c.smax + zero)
    sat = soil / c.smax
    runoff = eff * sat.clamp(min=0.) ** c.gamma
    aet = torch.minimum(soil_pet, (c.max_pet - evap) * sat)
    wet = _tiny(soil + eff - aet - runoff)
    aet = aet + wet.clamp(max=0.)
    wet = wet.clamp(min=0.)
    runoff = runoff * c.cfa
    recharge = torch.minimum(c.rgmax + zero, c.fg * runoff)
    pot = where(c.arid_gw & (prec <= c.pcrit), recharge, zero)
    recharge = recharge - pot
    runoff = runoff - pot
    wet = wet + pot / c.cfa
    over_thaw = (over + (wet - c.smax).clamp(min=0.)) * c.cfa
    wet = torch.minimum(wet, c.smax + zero)
    total = where(thawed, runoff + immediate * c.cfa + over_thaw, over * c.cfa + eff * c.cfa)
    soil = where(thawed, wet, soil)
    recharge, aet = where(thawed, recharge, zero), where(thawed, aet, zero)
    change = change + soil - before
    cell_aet = (change - prec) * (c.cfa - 1.) + (aet + evap + snow_evap) * c.cfa
    total = (total + cell_aet.clamp(max=0.)).clamp(min=0.)
    short = (total - recharge).clamp(max=0.)
    soil, used = soil + short, torch.minimum(recharge, total)
    on = lambda x: where(land, x, zero)  # noqa: E731
    c.canopy.copy_(on(canopy))
    c.soil.copy_(on(soil))
    share = laf / c.cont
    grids = dict(prec=prec, temp=T + zero, pet=pet, aet=on(aet) * share, swe=c.snow * share, soil_wc=c.soil * share,
                 runoff=on(total) * share, gw_recharge=on(used) * share)
    return on(total - used), on(recharge), transfer, prec, open_pet, grids


def _shrink(S, most, half, evx):
    return (1. - ((S - most).abs() * (0.5 if half else 1.) / most) ** evx).clamp(0., 1.)


def _routing(c, v, up, month_start):
    """One day of routing (routing.cpp:1835-4520): the transported volume and the
    evaporation of the water bodies; month_start: the month that the day begins
    (1 to 12), else 0."""
    where = torch.where
    rs, recharge, transfer, owp, owpet, _ = v
    zero = torch.zeros_like(rs)
    to_km3 = c.area * 1e-8
    runoff = where(c.laf <= 0, transfer * to_km3 * c.laf_prev, rs * to_km3 * c.laf)
    into = recharge * to_km3 * c.laf
    eg = torch.exp(-c.kg)
    gw = _tiny(c.gw * eg + into / c.kg * (1. - eg))
    base = c.gw - gw + into
    dry = base <= 0
    gw, base = where(dry, _tiny(c.gw + into), gw), where(dry, zero, base)
    c.gw.copy_(gw)
    flow, direct = runoff + base, zero
    if c.frac:
        split = ~c.sink
        kept = where(c.arid, zero, c.fcatch * base)
        direct = where(split, (1. - c.fcatch) * runoff + base - kept, zero)
        flow = where(split, c.fcatch * runoff + kept, flow)
    a6, out, owe = c.area / 1e6, zero, zero

    def demand(rf):
        return ((1. - c.cfa) * owp * rf + c.cfa * owpet * rf).clamp(min=0.)

    def keep(has, name, value):
        getattr(c, name).copy_(where(has, value, getattr(c, name)))

    # local lake (routing.cpp:2318-2490)
    has, S0, most = c.has_ll, c.loclake, where(c.has_ll, c.max_ll, 1. + 0. * c.max_ll)
    gain, pet = flow + owp * c.rf_loclake * a6 * c.ll, demand(c.rf_loclake) * a6 * c.ll
    avail = S0 + most + gain
    S = where(pet > avail.clamp(min=0.), -most + zero, S0 + gain - pet)
    q = where(S0 > 0, c.ks * S0 * (S0 / most).clamp(min=0.) ** 1.5, zero)
    q = where(S <= 0, zero, torch.minimum(q, S))
    S = _tiny(S - q)
    q, S = q + (S - most).clamp(min=0.), torch.minimum(S, most + zero)
    owe = owe + where(has, torch.minimum(pet, avail.clamp(min=0.)), zero)
    keep(has, "rf_loclake", _shrink(S, most, True, c.evx))
    keep(has, "loclake", S)
    flow = where(has, q, flow)
    # local wetland (routing.cpp:2495-2617)
    has, S0, most = c.has_lw, c.locwetl, where(c.has_lw, c.max_lw, 1. + 0. * c.max_lw)
    gain, pet = flow + owp * c.rf_locwetl * a6 * c.lw, demand(c.rf_locwetl) * a6 * c.lw
    avail = S0 + gain
    S = _tiny(where(pet > avail, zero, avail - pet))
    q = where(S > 0, torch.minimum(c.ks * S * (S / most).clamp(min=0.) ** 2.5, S), zero)
    S = S - q
    q, S = q + (S - most).clamp(min=0.), torch.minimum(S, most + zero)
    owe = owe + where(has, torch.minimum(pet, avail), zero)
    keep(has, "rf_locwetl", _shrink(S, most, False, c.evx))
    keep(has, "locwetl", S)
    flow = where(has, q, flow) + up
    # global lake (routing.cpp:2630-2804)
    has, S0, most = c.has_gl, c.glolake, where(c.has_gl, c.max_gl, 1. + 0. * c.max_gl)
    es = torch.exp(-c.ks)
    gain = flow + owp * c.la6
    pet = ((1. - c.cfa) * owp + c.cfa * owpet * c.rf_glolake).clamp(min=0.) * c.la6
    avail = gain + most + S0
    S = S0 * es + (gain - pet) / c.ks * (1. - es)
    q = gain + S0 - S - pet
    q, S = q + (S - most).clamp(min=0.), torch.minimum(S, most + zero)
    S, q = where(q < 0, S0 + gain - pet, S), q.clamp(min=0.)
    dry = pet > avail
    S, q = _tiny(where(dry, -most + zero, S)), where(dry, zero, q)
    owe = owe + where(has, torch.minimum(pet, avail), zero)
    keep(has, "rf_glolake", _shrink(S, most, True, c.evx))
    keep(has, "glolake", S)
    flow = where(has, q, flow)
    # reservoir (routing.cpp:2807-3082)
    has, S0, most = c.has_res, c.res, where(c.has_res, c.max_res, 1. + 0. * c.max_res)
    gain = flow + owp * c.ra6
    pet = ((1. - c.cfa) * owp + c.cfa * (owpet * c.rf_res)).clamp(min=0.) * c.ra6
    avail = S0 + gain
    S = _tiny(avail - torch.minimum(pet, avail))
    low = S < most * 0.1
    keep(has & (c.start == month_start), "k_release", where(low, 0.1 + zero, S / (most * 0.85)))
    c4 = 4. * c.c_ratio * c.c_ratio
    q = where(c.c_ratio >= 0.5, c.k_release * c.release, c4 * c.k_release * c.release + (1. - c4) * flow * 1e9 / 86400.)
    q = (where(low, 0.1 * q, q) * 86400. / 1e9).clamp(min=0.)
    S = S - q
    q, S = q + (S - most).clamp(min=0.), torch.minimum(S, most + zero)
    q, S = q + S.clamp(max=0.), S.clamp(min=0.)
    owe = owe + where(has, torch.minimum(pet, avail), zero)
    keep(has, "rf_res", _shrink(S, most, False, 2.81383 + 0. * c.evx))
    keep(has, "res", S)
    flow = where(has, q, flow)
    # global wetland (routing.cpp:3178-3297)
    has, S0, most = c.has_gw, c.glowetl, where(c.has_gw, c.max_gw, 1. + 0. * c.max_gw)
    gain, pet = flow + owp * c.rf_glowetl * a6 * c.gw_pct, demand(c.rf_glowetl) * a6 * c.gw_pct
    avail = gain + S0
    S = S0 * es + (gain - pet) / c.ks * (1. - es)
    q = avail - S - pet
    dry = pet > avail
    S, q = where(dry, zero, S), where(dry, zero, q)
    q, S = q + (S - most).clamp(min=0.), _tiny(torch.minimum(S, most + zero))
    owe = owe + where(has, torch.minimum(pet, avail), zero)
    keep(has, "rf_glowetl", _shrink(S, most, False, c.evx))
    keep(has, "glowetl", S)
    flow = where(has, q, flow)
    # river (routing.cpp:3385-3514, 7274-7341)
    flow = flow + direct
    S0 = c.river
    if c.velo == 0:
        v_river = c.default_velocity + zero
    else:
        if c.velo == 1:
            depth = 0.349 * (flow * (1e9 / 86400.)).clamp(min=0.) ** 0.341
            area = depth * (2. * depth + c.bw)
        else:
            area = S0 / c.length * 1e6
            depth = -c.bw / 4. + torch.sqrt(c.bw * c.bw / 16. + 0.5 * area)
        hr = area / (c.bw + 2. * math.sqrt(5.) * depth)
        v_river = (c.mr * hr.clamp(min=0.) ** (2. / 3.) * c.slope * 86.4).clamp(min=0.00001)
    K = v_river / c.length
    eK, omeK = torch.exp(-K), -torch.expm1(-K)
    most = flow + K * S0 * eK / omeK
    S = _tiny(where(most < 0, zero, S0 * eK + flow * omeK / K))
    out = (flow + S0 - where(most < 0, most, S)).clamp(min=0.)
    c.river.copy_(S)
    # the land fraction of the next day (routing.cpp:5034-5188, 5343-5352)
    f = sum(where(has, rf.clamp(min=0.) * pct, zero) for has, rf, pct in
            ((c.has_ll, c.rf_loclake, c.ll), (c.has_lw, c.rf_locwetl, c.lw), (c.has_gw, c.rf_glowetl, c.gw_pct)))
    body = c.has_ll | c.has_lw | c.has_gw
    laf = where(body, (c.laf - (f - c.fswb) * 100.).clamp(min=0.), c.laf)
    c.fswb.copy_(where(body, f, c.fswb))
    c.laf_prev.copy_(c.laf)
    c.laf.copy_(laf)
    c.started.fill_(1.)
    return out, owe


@torch.no_grad()
def _simulate(region, weather, case, seed):
    dev, days, members = _device(), case["days"], case["members"]
    pf, gf = _members(case, seed)
    offset = _offsets(region)
    order = np.argsort(offset, kind="stable")
    rank = np.empty_like(order)
    rank[order] = np.arange(order.size)
    start = np.searchsorted(offset[order], np.arange(offset.max() + 2))
    c = _constants(region, order, dev, members, gf)
    P, T, S = (torch.as_tensor(np.ascontiguousarray(w[:, order]), device=dev) for w in weather)
    pf = torch.ones(1, device=dev, dtype=torch.float32) if pf is None else torch.as_tensor(pf, device=dev)
    n = region.ncell
    down = np.where(region.downstream < 0, n, rank[np.maximum(region.downstream, 0)])[order]
    down = torch.as_tensor(down, device=dev)
    stations = _stations(case, region)
    at = rank[stations]                       # sorted position of each station
    # stations by sorted position, so that those of some cells are one range
    st_sort = np.argsort(at, kind="stable")
    at_sorted = at[st_sort]
    q_all = torch.zeros((days, stations.size, members), device=dev, dtype=torch.float64)
    at_dev = torch.as_tensor(at_sorted, device=dev)
    months = _months(days)
    grids = {k: torch.zeros((months[-1] + 1, n), device=dev, dtype=torch.float64) for k in GRIDS} \
        if case["option"] == "grids" else {}
    q_prev, prev = None, (0, 0)
    nlevel = int(offset.max()) + 1
    off = torch.as_tensor(offset[order], device=dev)
    month = torch.as_tensor(months, device=dev)
    first = torch.zeros(367, device=dev, dtype=torch.float64)   # day of the year -> month that it begins, from 1
    first[list(FIRST)] = torch.arange(1., 13., device=dev, dtype=torch.float64)
    for t in range(days + nlevel - 1):
        up = torch.zeros((n + 1, members), device=dev, dtype=torch.float64)
        if q_prev is not None:
            up.index_add_(0, down[prev[0]:prev[1]], q_prev)
        lo, hi = int(start[max(0, t - days + 1)]), int(start[min(nlevel - 1, t) + 1])
        g, d, cell = c.cut(lo, hi), t - off[lo:hi], torch.arange(lo, hi, device=dev)
        w = [x[d, cell].double()[:, None] for x in (P, T, S)]
        w[0] = w[0] * pf.double()[None, :]
        doy = (DOY0 - 1 + d) % 365 + 1
        v = _vertical(g, *w, doy.double()[:, None])
        q, owe = _routing(g, v, up[lo:hi], first[doy][:, None])
        if grids:
            term = v[5]
            term["river_avail"] = torch.where(g.sink, 0. * q, q)
            term["cell_runoff"] = term["river_avail"] - up[lo:hi]
            term["storage"] = sum(getattr(g, k) for k in ("gw", "river", "loclake", "locwetl", "glolake", "glowetl",
                                                          "res"))
            term["open_water_evap"] = (owe + torch.where(g.sink, q, 0. * q)) * 1e8 / (g.area * g.cont)
            for k in GRIDS:
                grids[k][month[d], cell] += term[k][:, 0]
        i, j = np.searchsorted(at_sorted, (lo, hi))
        q_all[t - off[at_dev[i:j]], torch.arange(i, j, device=dev)] = q[at_dev[i:j] - lo]
        q_prev, prev = q, (lo, hi)
    inv = np.empty_like(st_sort)
    inv[st_sort] = np.arange(st_sort.size)
    back = torch.as_tensor(rank, device=dev)
    names = dict(laf_started="started", fswb_next="fswb")
    state = {}
    if members == 1:
        for k in STATE:
            if k == "snow_band":
                state[k] = c.band[:, back, 0].T.contiguous().reshape(-1).cpu().numpy()
            else:
                state[k] = getattr(c, names.get(k, k))[back, 0].cpu().numpy()
    return q_all[:, inv].cpu().numpy(), state, {k: g[:, back].cpu().numpy() for k, g in grids.items()}
