"""The timed workloads of the column radiation: what a user's model has this package do, through its public calls.

A case is one radiation request (or a batch, or the whole radiation call): ``listed()`` gives the fixed set,
``draw(rng)`` one more from the same ranges, ``prepare(case, seed)`` the solver handle and the device-resident
column state a model holds before the call, ``run(state)`` one pass, and ``exact(case, seed)`` the same outputs in
64-bit arithmetic: a plain torch restatement of RRTMG's longwave and shortwave column solve (set-up, cloud optics,
the k-distribution gas optics of the 16 + 14 bands, rtrnmr / rtrn / rtrnmc and spcvrtc with the adding method),
reading only the packed coefficient tables.

Columns are synthetic with the distributions of woof_nam_b200.columns (its docstring states the rules), formed on
the GPU from the seed so that new inputs cost little.
"""
from __future__ import annotations

import math
from functools import lru_cache
from pathlib import Path

import numpy as np
import torch

DEV = "cuda" if torch.cuda.is_available() else "cpu"
SOLCON = 1368.22
LW_FLOP, SW_FLOP = 716013.0, 1784199.0     # counted operations per 61-layer column / sunlit column


# ----------------------------------------------------------------------------------------------- the cases
def _case(name=None, **kw):
    c = {"kind": "solve", "sizes": "1024", "nlay": 61, "route": "nam", "parts": "both", "clouds": "water",
         "aerosol": False, "sun": "mixed", "iovrlw": 1, "iswmode": 2, "profiles": False, "lw_chunk": 0,
         "sw_sweep_chunk": 0}
    c.update(kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # a single-column model's daytime step: nothing but launch latency and one column's dependency chain
        _case("column_1", sizes="1", sun="day"),
        # the plain 1,024-column request (about one 954-point row of the 12 km grid): a few columns per SM
        _case("plain_1024", sizes="1024"),
        # a ragged window of a 40-layer model with random cloud overlap and the discrete-ordinates two-stream
        _case("ragged_4999_random_40lay", sizes="4999", nlay=40, iovrlw=0, iswmode=3),
        # the 180 x 180 3 km nest, both solves, default configuration
        _case("nest_180x180", sizes="32400"),
        # a longwave-only radiation step (lslwr without lsswr) of the 333 x 333 nest
        _case("lw_step_333x333", sizes="110889", parts="lw"),
        # a shortwave-only step of a fully sunlit domain, odd column count
        _case("sw_step_day_50021", sizes="50021", parts="sw", sun="day"),
        # the three nests as one batched request
        _case("nests_batch", sizes="110889,270000,32400"),
        # the 12 km parent grid, 954 x 835, the tiles the tuner picks for it
        _case("parent_954x835", sizes="796590", lw_chunk=131072, sw_sweep_chunk=65536),
        # cloud optical properties given directly (the diagnostic input form): thick, near-conservative clouds
        # under a low sun, 200,000 columns
        _case("direct_optics_200k", sizes="200000", clouds="direct", sun="low"),
        # a nest with aerosol optics on the request
        _case("aerosol_180x180", sizes="32400", aerosol=True),
        # the McICA route with the band heating and flux profiles asked for, eight rows of the parent grid
        _case("mcica_profiles_7632", sizes="7632", route="mcica", profiles=True),
        # the whole radiation call (grrad's set-up, gases, ozone, aerosol climatology, clouds, surface, solve)
        # of a 180 x 180 domain
        _case("radiation_call_180x180", kind="call", sizes="32400"),
    ]


def draw(rng):
    n = int(round(math.exp(rng.uniform(0.0, math.log(400000.0)))))
    kind = rng.choice(["both", "both", "both", "lw", "sw", "batch", "direct", "aerosol", "mcica", "random"])
    kw = {"nlay": rng.choice([40, 61, 61, 64, rng.randint(30, 64)]), "iswmode": rng.choice([2, 2, 3]),
          "sun": rng.choice(["mixed", "mixed", "day"])}
    if kind in ("lw", "sw"):
        kw["parts"] = kind
    elif kind == "batch":
        k = rng.randint(2, 6)
        cuts = sorted(rng.uniform(0.0, 1.0) for _ in range(k - 1))
        w = [b - a for a, b in zip([0.0] + cuts, cuts + [1.0])]
        return _case(sizes=",".join(str(max(1, int(n * x))) for x in w), **kw)
    elif kind == "direct":
        kw.update(clouds="direct", sun="low")
    elif kind == "aerosol":
        kw["aerosol"], n = True, min(n, 100000)
    elif kind == "mcica":
        kw["route"], kw["profiles"] = "mcica", n < 20000
    elif kind == "random":
        kw["iovrlw"] = 0
    return _case(sizes=str(n), **kw)


def _sizes(case):
    return [int(x) for x in case["sizes"].split(",")]


# ---------------------------------------------------------------------------------------------- the inputs
def _columns(n, seed, case):
    """One request's column state on the device: float32, [field][level][column], level 0 the model top."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    f64 = dict(dtype=torch.float64, device=DEV)

    def uni(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=g, **f64)

    nm = case["nlay"] - 1
    direct = case["clouds"] == "direct"
    ps = uni(950.0, 1030.0, n)
    s = (torch.arange(nm + 1, **f64) / nm) ** 1.4
    st = (300.0 - 2.0) / (1000.0 - 2.0)
    a = torch.where(s < st, 2.0 + 298.0 * s / st, torch.full_like(s, 300.0))
    b = torch.where(s < st, torch.zeros_like(s), (s - st) / (1.0 - st))
    pi = a[:, None] + b[:, None] * (ps[None, :] - 300.0)
    if direct:
        pi[1] = 2.1
    pl = 0.5 * (pi[:-1] + pi[1:])
    ts = 288.0 + 5.0 * torch.randn(n, generator=g, **f64)
    t = ts[None] * (pl / ps[None]) ** (287.04 * 0.0065 / 9.80665)
    t = torch.where(pl < 200.0, torch.full_like(t, 217.0), t.clamp(min=217.0))
    rh = uni(0.1, 0.95, nm, n)
    tc = t - 273.15
    es = torch.minimum(6.112 * torch.exp(17.67 * tc / (tc + 243.5)), 0.5 * pl)
    q = rh * 0.622 * es / (pl - 0.378 * es)
    q = torch.where(pl < 200.0, q.clamp(max=3.0e-6), q).clamp(min=1.0e-7)

    def ozone(p):
        return (8.0e-6 * torch.exp(-torch.log(p / 10.0) ** 2 / 2.88)).clamp(min=0.03e-6) * (47.9982 / 28.9644)

    plvl = torch.cat([torch.full((1, n), 1.0e-6, **f64), pi])
    plyr = torch.cat([0.5 * plvl[1:2], pl])
    tlyr = torch.cat([t[:1], t])
    tskin = tlyr[-1] + 3.0 * torch.randn(n, generator=g, **f64)
    lpl, lly = torch.log(plvl[1:-1]), torch.log(plyr)
    tlvl = torch.cat([tlyr[:1], tlyr[1:] + (tlyr[:-1] - tlyr[1:]) * (lpl - lly[1:]) / (lly[:-1] - lly[1:]),
                      tskin[None]])
    cf = ((rh - 0.8) / 0.2).clamp(0.0, 1.0)
    nlay = nm + 1
    clouds = torch.zeros(9, nlay, n, dtype=torch.float32, device=DEV)
    clouds[0, 1:] = cf
    if direct:
        tau = torch.exp(uni(math.log(0.1), math.log(500.0), nm, n))
        for k, v in ((1, tau), (2, uni(1.0 - 1.0e-7, 1.0, nm, n)), (3, torch.full_like(cf, 0.85))):
            clouds[k, 1:] = torch.where(cf > 0, v, torch.zeros_like(v))
    else:
        fl = ((t - 253.0) / 20.0).clamp(0.0, 1.0)
        for k, share, median, reff in ((1, fl, 50.0, 10.0), (3, 1.0 - fl, 20.0, 50.0)):
            w = cf * share
            col = median * torch.exp(torch.randn(n, generator=g, **f64))
            tot = w.sum(0)
            path = torch.where(tot > 0, col / tot.clamp(min=1e-300), torch.zeros_like(tot))[None] * share
            clouds[k, 1:] = torch.where(w > 0, path, torch.zeros_like(path))
            clouds[k + 1, 1:] = reff
    lo, hi = {"mixed": (-1.0, 1.0), "day": (0.05, 1.0), "low": (0.01, 0.05)}[case["sun"]]
    gas = torch.tensor([420.0e-6, 0.31e-6, 1.50e-6, 0.209, 1.50e-8, 3.520e-10, 6.358e-10, 1.500e-10, 1.397e-10,
                        8.2000e-11], dtype=torch.float32, device=DEV)
    d = {"plyr": plyr, "plvl": plvl, "tlyr": tlyr, "tlvl": tlvl, "qlyr": torch.cat([q[:1], q]),
         "olyr": ozone(plyr), "gasvmr": gas[:, None, None].expand(10, nlay, n), "clouds": clouds,
         "sfcemis": uni(0.95, 1.0, n), "tsfg": tskin, "sfcalb": uni(0.06, 0.8, n)[None].expand(4, n),
         "coszen": uni(lo, hi, n)}
    if case["aerosol"]:
        # optical depth falling off with pressure, absorbing to conservative, forward scattering
        amt = torch.exp(0.8 * torch.randn(n, generator=g, **f64))[None] * (plyr / plvl[-1:]) ** 2
        for key, nb, scale in (("faersw", 14, 0.008), ("faerlw", 16, 0.002)):
            f = torch.empty(3, nb, nlay, n, dtype=torch.float32, device=DEV)
            for band in range(nb):
                f[0, band] = amt * scale * (0.5 + band / nb)
            f[1] = 0.3 + 0.69 * torch.rand(nb, nlay, n, generator=g, dtype=torch.float32, device=DEV)
            f[2] = 0.5 + 0.25 * torch.rand(nb, nlay, n, generator=g, dtype=torch.float32, device=DEV)
            d[key] = f
    return {k: v.to(torch.float32).contiguous() for k, v in d.items()}


def _config(case):
    from woof_nam_b200.solver import SolverConfig
    p = case["profiles"]
    return SolverConfig(nlay=case["nlay"], route=case["route"], parts=case["parts"], iswmode=case["iswmode"],
                        diagnostic=case["clouds"] == "direct", iovrlw=case["iovrlw"], lw_chunk=case["lw_chunk"],
                        sw_sweep_chunk=case["sw_sweep_chunk"], lhlw0=p, lhlwb=p, lhsw0=p, lhswb=p, lflxprf=p)


CALL = dict(solhr=18.5, dtswav=1200.0 / 3600.0, nrads=48, kmonsav=7, k1oz=6, k2oz=7, facoz=0.4, ico2flg=2,
            ialbflg=1, iemslw=1)


def _prepare_call(case, seed):
    """A domain's model state, surface and cloud fields, and the climatologies of its month."""
    from woof_nam_b200 import aerosols, solar
    from woof_nam_b200.columns import cloud_state, front_tables, make_columns, model_state, surface_state
    from woof_nam_b200.grrad import layers
    from woof_nam_b200.solver import RadSolver
    n = _sizes(case)[0]
    im = math.isqrt(n)
    n = im * im
    solver = RadSolver(_config(case))

    def dev(a):
        return torch.as_tensor(np.ascontiguousarray(a), device="cuda")

    model = model_state(make_columns(n, seed))
    lay = {k: v.cpu().numpy() for k, v in layers(solver, {k: dev(v) for k, v in model.items()}).items()}
    state = dict(model)
    cld = cloud_state(lay, seed + 1)
    state.update({k: cld[k] for k in ("clw", "f_ice", "f_rain", "r_rime", "cldfk1")})
    lon = np.linspace(-2.4, -0.9, im, dtype=np.float32)[None, :].repeat(im, 0).ravel()
    lat = np.linspace(0.2, 1.1, im, dtype=np.float32)[:, None].repeat(im, 1).ravel()
    state.update(surface_state(n, seed + 2))
    state.update(glon=lon, glat=lat, sinlat=np.sin(lat), coslat=np.cos(lat))
    tab = front_tables(seed + 3)
    clim = {k: dev(v) if isinstance(v, np.ndarray) else v for k, v in tab.items()}
    clim["co2_glb"] = dev(np.atleast_1d(np.float32(tab["co2_glb"])))
    return {"kind": "call", "solver": solver, "state": {k: dev(v) for k, v in state.items()}, "clim": clim,
            "sun": solar.sol_update((2026, 7, 1, 18, 30, 0), deltsw=1200.0, deltim=25.0), "im": im,
            "aerosols": aerosols.Aerosols(solver, 7), "work": None, "out": None}


def prepare(case, seed):
    if case["kind"] == "call":
        return _prepare_call(case, seed)
    from woof_nam_b200.solver import RadSolver
    solver = RadSolver(_config(case))
    cols = [_columns(n, seed + 1000003 * r, case) for r, n in enumerate(_sizes(case))]
    return {"kind": "solve", "solver": solver, "cols": cols,
            "outs": [solver.alloc_outputs(int(c["tsfg"].shape[0])) for c in cols]}


def run(state):
    if state["kind"] == "call":
        from woof_nam_b200.chain import radiation_call
        res = radiation_call(state["solver"], state["state"], state["clim"], sun=state["sun"], im=state["im"],
                             aerosols=state["aerosols"], work=state["work"], out=state["out"], **CALL)
        state["work"] = res.pop("work")
        state["out"] = res
        return res
    if len(state["cols"]) == 1:
        return state["solver"].solve(state["cols"][0], SOLCON, out=state["outs"][0])
    return state["solver"].solve_batch(state["cols"], [SOLCON] * len(state["cols"]), outs=state["outs"])


def work(case):
    nlay, n = case["nlay"], sum(_sizes(case))
    lw, sw = case["parts"] != "sw", case["parts"] != "lw"
    day = {"mixed": 0.5, "day": 1.0, "low": 1.0}[case["sun"]]
    words = 24 * nlay + 1 + 3 + (lw * (nlay + 3)) + (sw * 5) + 1        # the inputs the parts read
    words += lw * (nlay + 6) + sw * (nlay + 13)                        # the heating rates and fluxes
    if case["aerosol"]:
        words += nlay * (lw * 32 + sw * 42)
    if case["profiles"]:
        words += lw * (17 * nlay + 4 * (nlay + 1)) + sw * (15 * nlay + 4 * (nlay + 1))
    if case["route"] == "mcica":
        words += 9 * nlay
    if case["kind"] == "call":
        words = 15 * nlay + 60 + 2 * nlay + 19                         # model, cloud and surface fields; outputs
    flops = n * (nlay / 61.0) * (lw * LW_FLOP + sw * day * SW_FLOP)
    return {"bytes": 4.0 * words * n, "flops": flops}


def tolerance(case):
    # Single-precision optics and transfer under an algorithm that looks its exponentials up in nearest-entry
    # tables: one entry step is 3e-4 of a layer's transmission, so a single value can differ by far more than the
    # 2-norm.  About four times what the float solve shows against exact(): 2-norm 3.1e-6 (heating of one band
    # 5.2e-6; near-conservative clouds under a low sun 2.6e-5), largest value 4.1e-4 (2.1e-3; 1.1e-3).  The
    # sub-column words of the McICA route are whole numbers and stay the same.
    direct = case["clouds"] == "direct"
    return {"rel": 1.0e-4 if direct else 2.0e-5,
            "max": 8.0e-3 if case["profiles"] else 4.0e-3 if direct else 2.0e-3, "differ": 0.0}


# -------------------------------------------------------------------------------- the solve in 64 bits (torch)
EXACT_COLUMNS = 120000                      # above this exact() would take more than about 20 seconds
EXACT_CHUNK = 4096


def f32(x):
    return float(np.float32(x))


@lru_cache(maxsize=1)
def _tables():
    import woof_nam_b200
    z = np.load(Path(woof_nam_b200.__file__).resolve().parent / "data" / "rrtm_tables.npz")
    return {k: torch.as_tensor(z[k].astype(np.float64), device=DEV) for k in z.files}


@lru_cache(maxsize=1)
def _luts():
    n = 10000
    i = np.arange(1, n, dtype=np.float64)
    bp = 1.0 / f32(0.278)
    ta = bp * (i / (n - i))
    lim = np.trunc(-math.log(np.finfo(np.float64).tiny))
    e = np.where(ta >= lim, f32(1e-20), np.exp(-ta))
    tfn = np.where(ta < f32(0.06), ta / 6.0, 1.0 - 2.0 * (1.0 / ta - e / (1.0 - e)))
    lw = [np.concatenate([[a], m, [b]]) for a, m, b in ((1.0, e, f32(1e-20)), (0.0, tfn, 1.0), (0.0, ta, f32(1e10)))]
    sw = np.concatenate([[1.0], np.exp(-(1.0 / 0.278) * (i / (n - i))), [f32(1e-20)]])
    return [torch.as_tensor(a, device=DEV) for a in lw + [sw]]


LW_NS = (0, 10, 22, 38, 52, 68, 76, 88, 96, 108, 114, 122, 130, 134, 136, 138, 140)
SW_NS = (0, 6, 18, 26, 34, 44, 54, 56, 66, 74, 80, 86, 94, 100, 112)


def _trunc(x):
    return x.to(torch.int64)


def _rows(t, ind):
    """Rows ind (1-based) of a [rows][g] table."""
    return t[(ind - 1).clamp(0, t.shape[0] - 1)]


def _lerp(t, ind, frac):
    a = _rows(t, ind)
    return a + frac[:, None] * (_rows(t, ind + 1) - a)


def _surface_first(cols, key, off=0):
    return cols[key].to(torch.float64).flip(off)


def _lw_points(cols, T):
    """Layer quantities of lwrad_prep and setcoef, [nlay][n], surface first."""
    plf, p, t = (_surface_first(cols, k) for k in ("plvl", "plyr", "tlyr"))
    q, o = _surface_first(cols, "qlyr"), _surface_first(cols, "olyr")
    gas = _surface_first(cols, "gasvmr", 1)
    dlp = plf[:-1] - plf[1:]
    h2o = (q * (28.9644 / 18.0154) / (1.0 - q)).clamp(min=0.0)
    tem0 = (1.0 - h2o) * 28.9644 + h2o * 18.0154
    dry = 1.0e-20 * 1.0e3 * 6.0221415e23 * dlp / (100.0 * 9.80665 * tem0 * (1.0 + h2o))
    tiny = 1.0e-12 * dry
    col = [(dry * h2o).clamp(min=0.0), torch.maximum(tiny, dry * gas[0]),
           torch.maximum(tiny, dry * (o * (28.9644 / 47.9982)).clamp(min=0.0)), torch.maximum(tiny, dry * gas[1]),
           torch.maximum(tiny, dry * gas[2]), (dry * gas[3]).clamp(min=0.0), (dry * gas[4]).clamp(min=0.0)]
    s = {"pav": p, "tav": t, "dry": dry, "dlp": dlp, "low": torch.log(p) > f32(4.56)}
    for m in range(7):
        s[f"c{m}"] = col[m]
    for m, gi in enumerate((8, 5, 6, 7)):
        s[f"w{m}"] = (dry * gas[gi]).clamp(min=0.0)
    s["brd"] = dry - sum(col[1:])
    h = col[0] / dry.clamp(min=f32(1e-30))
    plog = torch.log(p)
    jp = _trunc(36.0 - 5.0 * (plog + f32(0.04))).clamp(1, 58)
    fp = (5.0 * (T["lw_preflog"][jp - 1] - plog)).clamp(0.0, 1.0)
    t1, t2 = (t - T["lw_tref"][jp - 1]) / 15.0, (t - T["lw_tref"][jp]) / 15.0
    jt, jt1 = _trunc(3.0 + t1).clamp(1, 4), _trunc(3.0 + t2).clamp(1, 4)
    ft, ft1 = (t1 - (jt - 3)).clamp(-0.5, 1.5), (t2 - (jt1 - 3)).clamp(-0.5, 1.5)
    s.update(jp=jp, jt=jt, jt1=jt1, f10=(1.0 - fp) * ft, f00=(1.0 - fp) * (1.0 - ft), f11=fp * ft1,
             f01=fp * (1.0 - ft1))
    forf = p * (f32(296.0) / f32(1013.0)) / (t * (1.0 + h))
    s["sm"] = p / t
    s["sn2"] = (p / t) * (s["brd"] / (dry + col[0]))
    tm = (t - f32(180.8)) / f32(7.2)
    s["im"] = _trunc(tm).clamp(1, 18)
    s["fm"] = tm - s["im"]
    lo = s["low"]
    a, b = (332.0 - t) / 36.0, (t - 188.0) / 36.0
    ifl = _trunc(a).clamp(1, 2)
    s["if"] = torch.where(lo, ifl, torch.full_like(ifl, 3))
    s["ff"] = torch.where(lo, a - ifl, b - 1.0)
    c = (t - 188.0) / f32(7.2)
    isl = (_trunc(c) - 7).clamp(1, 9)
    s["is"] = torch.where(lo, isl, torch.ones_like(isl))
    s["fs"] = torch.where(lo, c - (isl + 7), torch.zeros_like(c))
    s["sfac"] = torch.where(lo, col[0] * h * forf, torch.zeros_like(c))
    s["ffac"] = col[0] * forf
    chi = T["lw_chi_mls"]

    def rat(i, a_, b_):
        return chi[i - 1, a_ - 1] / chi[i - 1, b_ - 1]

    for side, j in ((0, jp), (1, jp + 1)):
        for r, (a_, b_) in enumerate(((1, 2), (1, 3), (1, 4), (1, 6), (4, 2), (3, 2))):
            s[f"r{side}{r}"] = rat(j, a_, b_)

    def adj(cc, tt, thr, off, ex):
        x = cc / tt
        return torch.where(x > thr, (off + (x - off).clamp(min=1e-300) ** f32(ex)) * tt, cc)

    ch2, ch4 = dry * chi[jp, 1], dry * chi[jp, 3]
    s["an2o"] = adj(col[3], ch4, 1.5, 0.5, 0.65)
    s["a6"] = adj(col[1], ch2, 3.0, 2.0, 0.77)
    s["a7"] = torch.where(lo, adj(col[1], ch2, 3.0, 3.0, 0.79), adj(col[1], ch2, 3.0, 2.0, 0.79))
    s["a8"] = adj(col[1], ch2, 3.0, 2.0, 0.65)
    s["a13"] = adj(col[1], dry * f32(3.55e-4), 3.0, 2.0, 0.68)
    return s


def _spec(c1, rat, c2, mult):
    sc = c1 + rat * c2
    sp = c1 / sc
    sm = mult * sp.clamp(max=1.0 - f32(1e-6))
    j = _trunc(sm)
    return sc, sp, 1 + j, sm - j


def _sel(br, fs, ind):
    """Weights and rows of the three-point species interpolation (branch 0 low, 1 high, 2 linear)."""
    p = torch.where(br == 0, fs - 1.0, -fs)
    p4 = p ** 4
    lin = br == 2
    k0 = torch.where(lin, 1.0 - fs, p4)
    k1 = torch.where(lin, fs, 1.0 - p - 2.0 * p4)
    k2 = torch.where(lin, torch.zeros_like(p), p + p4)
    off = torch.tensor([[0, 9, 1, 10, 2, 11], [1, 10, 0, 9, -1, 8], [0, 9, 1, 10, 0, 0]], device=ind.device)[br]
    return (k0, k1, k2), ind[:, None] + off


def _major(s, A, q0, q1, joint):
    """The binary-species major absorption of a lower-atmosphere band; q = (sc, sp, js, fs) at both levels."""
    def br(sp, sq):
        return torch.where((sp < 0.125) & (sq < 0.125), 0, torch.where((sp > 0.875) & (sq > 0.875), 1, 2))
    b0 = br(q0[1], q1[1] if joint else q0[1])
    b1 = b0 if joint else br(q1[1], q1[1])
    out = 0.0
    for q, b, ind, fa, fb in ((q0, b0, ((s["jp"] - 1) * 5 + (s["jt"] - 1)) * 9, s["f00"], s["f10"]),
                              (q1, b1, (s["jp"] * 5 + (s["jt1"] - 1)) * 9, s["f01"], s["f11"])):
        (k0, k1, k2), ids = _sel(b, q[3], ind + q[2])
        acc = 0.0
        for i, k in enumerate((k0, k1, k2)):
            acc = acc + (k * fa)[:, None] * _rows(A, ids[:, 2 * i]) + (k * fb)[:, None] * _rows(A, ids[:, 2 * i + 1])
        out = out + q[0][:, None] * acc
    return out


def _bilin(s, B, q0, q1):
    """The binary-species major absorption of an upper-atmosphere band (five species points)."""
    out = 0.0
    for q, ind, fa, fb in ((q0, ((s["jp"] - 13) * 5 + (s["jt"] - 1)) * 5, s["f00"], s["f10"]),
                           (q1, ((s["jp"] - 12) * 5 + (s["jt1"] - 1)) * 5, s["f01"], s["f11"])):
        i, fs = ind + q[2], q[3]
        out = out + q[0][:, None] * (((1 - fs) * fa)[:, None] * _rows(B, i) + ((1 - fs) * fb)[:, None] * _rows(B, i + 5) +
                                     (fs * fa)[:, None] * _rows(B, i + 1) + (fs * fb)[:, None] * _rows(B, i + 6))
    return out


def _single(s, A, low):
    d = 1 if low else 13
    i0 = (s["jp"] - d) * 5 + (s["jt"] - 1) + 1
    i1 = (s["jp"] - d + 1) * 5 + (s["jt1"] - 1) + 1
    return (s["f00"][:, None] * _rows(A, i0) + s["f10"][:, None] * _rows(A, i0 + 1) +
            s["f01"][:, None] * _rows(A, i1) + s["f11"][:, None] * _rows(A, i1 + 1))


def _minor2(t, s, j, fj):
    """Bilinear minor-gas coefficient from t[temperature][species][g]."""
    m, f = s["im"] - 1, fj[:, None]
    a = t[m, j - 1] + f * (t[m, j] - t[m, j - 1])
    b = t[m + 1, j - 1] + f * (t[m + 1, j] - t[m + 1, j - 1])
    return a + s["fm"][:, None] * (b - a)


def _lw_gas(s, T, low):
    """taug, fracs [points][140] of the points in the lower (low) or upper atmosphere."""
    chi, chd = T["lw_chi_mls"], T["lw05_chi_mls_f64"]
    r = lambda lev, a, b, c=chi: float(c[lev - 1, a - 1] / c[lev - 1, b - 1])   # noqa: E731
    X = lambda k: s[k][:, None]                                                  # noqa: E731
    P = s["pav"].shape[0]
    tau, fr = [], []

    def tb(b, k):
        return T[f"lw{b:02d}_{k}"]

    def self_(b):
        return X("sfac") * _lerp(tb(b, "selfref"), s["is"], s["fs"])

    def for_(b):
        return X("ffac") * _lerp(tb(b, "forref"), s["if"], s["ff"])

    def mnr(b, k):
        return _lerp(tb(b, k), s["im"], s["fm"])

    def flat(b, k):
        return tb(b, k)[None].expand(P, -1)

    c = [s[f"c{m}"] for m in range(7)]

    def two(x1, x2, rate, mult):
        return _spec(x1, s[f"r0{rate}"], x2, mult), _spec(x1, s[f"r1{rate}"], x2, mult)

    def frac(b, key, x1, rat, x2, mult):
        _, _, j, f = _spec(x1, rat, x2, mult)
        return _lerp(tb(b, key), j, f)

    for b in range(1, 17):
        ng = LW_NS[b] - LW_NS[b - 1]
        zero = torch.zeros(P, ng, dtype=torch.float64, device=c[0].device)
        if b == 1:
            n2 = (s["brd"] * s["sn2"])[:, None]
            if low:
                cor = torch.where(s["pav"] < 250, 1 - f32(0.15) * (250 - s["pav"]) / f32(154.4), torch.ones_like(c[0]))
                g = cor[:, None] * (X("c0") * _single(s, tb(1, "absa"), 1) + self_(1) + for_(1) + n2 * mnr(1, "ka_mn2"))
            else:
                cor = 1 - f32(0.15) * (s["pav"] / f32(95.6))
                g = cor[:, None] * (X("c0") * _single(s, tb(1, "absb"), 0) + for_(1) + n2 * mnr(1, "kb_mn2"))
            f = flat(1, "fracrefa" if low else "fracrefb")
        elif b == 2:
            if low:
                cor = 1 - f32(0.05) * (s["pav"] - 100) / 900
                g = cor[:, None] * (X("c0") * _single(s, tb(2, "absa"), 1) + self_(2) + for_(2))
            else:
                g = X("c0") * _single(s, tb(2, "absb"), 0) + for_(2)
            f = flat(2, "fracrefa" if low else "fracrefb")
        elif b in (3, 4):
            if low:
                q0, q1 = two(c[0], c[1], 0, 8.0)
                g = _major(s, tb(b, "absa"), q0, q1, False) + self_(b) + for_(b)
                if b == 3:
                    _, _, j, fj = _spec(c[0], r(3, 1, 2), c[1], 8.0)
                    g = g + X("an2o") * _minor2(tb(3, "ka_mn2o"), s, j, fj)
                f = frac(b, "fracrefa", c[0], r(9, 1, 2) if b == 3 else r(11, 1, 2), c[1], 8.0)
            else:
                x1 = c[0] if b == 3 else c[2]
                q0, q1 = two(x1, c[1], 0 if b == 3 else 5, 4.0)
                g = _bilin(s, tb(b, "absb"), q0, q1)
                if b == 3:
                    _, _, j, fj = _spec(c[0], r(13, 1, 2), c[1], 4.0)
                    g = g + for_(3) + X("an2o") * _minor2(tb(3, "kb_mn2o"), s, j, fj)
                else:
                    g = g * torch.tensor([1.0] * 7 + [f32(v) for v in (0.92, 0.88, 1.07, 1.1, 0.99, 0.88, 0.943)],
                                         dtype=torch.float64, device=g.device)
                f = frac(b, "fracrefb", x1, r(13, 1, 2) if b == 3 else r(13, 3, 2), c[1], 4.0)
        elif b == 5:
            xs = X("w0") * flat(5, "ccl4")
            if low:
                q0, q1 = two(c[0], c[1], 0, 8.0)
                _, _, j, fj = _spec(c[0], f32(r(7, 1, 2, chd)), c[1], 8.0)
                g = (_major(s, tb(5, "absa"), q0, q1, True) + self_(5) + for_(5) +
                     _minor2(tb(5, "ka_mo3"), s, j, fj) * X("c2") + xs)
                f = frac(5, "fracrefa", c[0], f32(r(5, 1, 2, chd)), c[1], 8.0)
            else:
                q0, q1 = two(c[2], c[1], 5, 4.0)
                g = _bilin(s, tb(5, "absb"), q0, q1) + xs
                f = frac(5, "fracrefb", c[2], f32(r(43, 3, 2, chd)), c[1], 4.0)
        elif b == 6:
            g = X("w1") * flat(6, "cfc11adj") + X("w2") * flat(6, "cfc12")
            if low:
                g = g + X("c0") * _single(s, tb(6, "absa"), 1) + self_(6) + for_(6) + X("a6") * mnr(6, "ka_mco2")
            f = flat(6, "fracrefa")
        elif b in (7, 9):
            x2, rate = (c[2], 1) if b == 7 else (c[4], 3)
            key, a = ("mco2", "a7") if b == 7 else ("mn2o", "an2o")
            if low:
                q0, q1 = two(c[0], x2, rate, 8.0)
                rm = r(3, 1, 3) if b == 7 else r(3, 1, 6)
                rp = r(3, 1, 3) if b == 7 else r(9, 1, 6)
                _, _, j, fj = _spec(c[0], rm, x2, 8.0)
                g = (_major(s, tb(b, "absa"), q0, q1, True) + self_(b) + for_(b) +
                     X(a) * _minor2(tb(b, "ka_" + key), s, j, fj))
                f = frac(b, "fracrefa", c[0], rp, x2, 8.0)
            else:
                g = x2[:, None] * _single(s, tb(b, "absb"), 0) + X(a) * mnr(b, "kb_" + key)
                if b == 7:
                    g = g * torch.tensor([1.0] * 5 + [f32(v) for v in (0.92, 0.88, 1.07, 1.1, 0.99, 0.855)] + [1.0],
                                         dtype=torch.float64, device=g.device)
                f = flat(b, "fracrefb")
        elif b == 8:
            g = X("w2") * flat(8, "cfc12") + X("w3") * flat(8, "cfc22adj")
            if low:
                g = (g + X("c0") * _single(s, tb(8, "absa"), 1) + self_(8) + for_(8) + X("a8") * mnr(8, "ka_mco2") +
                     X("c2") * mnr(8, "ka_mo3") + X("c3") * mnr(8, "ka_mn2o"))
            else:
                g = (g + X("c2") * _single(s, tb(8, "absb"), 0) + X("a8") * mnr(8, "kb_mco2") +
                     X("c3") * mnr(8, "kb_mn2o"))
            f = flat(8, "fracrefa" if low else "fracrefb")
        elif b in (10, 11, 14):
            cc = X("c1") if b == 14 else X("c0")
            g = cc * _single(s, tb(b, "absa" if low else "absb"), low)
            if low:
                g = g + self_(b)
            if low or b != 14:
                g = g + for_(b)
            if b == 11:
                g = g + (s["c5"] * s["sm"])[:, None] * mnr(11, "ka_mo2" if low else "kb_mo2")
            f = flat(b, "fracrefa" if low else "fracrefb")
        elif b in (12, 16):
            if low:
                x2, rate = (c[1], 0) if b == 12 else (c[4], 3)
                q0, q1 = two(c[0], x2, rate, 8.0)
                g = _major(s, tb(b, "absa"), q0, q1, True) + self_(b) + for_(b)
                f = frac(b, "fracrefa", c[0], r(10, 1, 2) if b == 12 else r(6, 1, 6), x2, 8.0)
            elif b == 12:
                g, f = zero, zero
            else:
                A = tb(16, "absb")
                g = X("c4") * ((s["f00"] + s["f01"])[:, None] * A[0] + (s["f10"] + s["f11"])[:, None] * A[1])
                f = flat(16, "fracrefb")
        elif b == 13:
            if low:
                q0, q1 = two(c[0], c[3], 2, 8.0)
                _, _, j, fj = _spec(c[0], r(1, 1, 4), c[3], 8.0)
                _, _, jc, fc = _spec(c[0], r(3, 1, 4), c[3], 8.0)
                g = (_major(s, tb(13, "absa"), q0, q1, True) + self_(13) + for_(13) +
                     X("a13") * _minor2(tb(13, "ka_mco2"), s, j, fj) + X("c6") * _minor2(tb(13, "ka_mco"), s, jc, fc))
                f = frac(13, "fracrefa", c[0], r(5, 1, 4), c[3], 8.0)
            else:
                g = X("c2") * mnr(13, "kb_mo3")
                f = flat(13, "fracrefb")
        else:   # 15
            if low:
                q0, q1 = two(c[3], c[1], 4, 8.0)
                rr = f32(r(1, 4, 2))
                _, _, j, fj = _spec(c[3], rr, c[1], 8.0)
                g = (_major(s, tb(15, "absa"), q0, q1, True) + self_(15) + for_(15) +
                     (s["brd"] * s["sm"])[:, None] * _minor2(tb(15, "ka_mn2"), s, j, fj))
                f = frac(15, "fracrefa", c[3], rr, c[1], 8.0)
            else:
                g, f = zero, zero
        tau.append(g)
        fr.append(f)
    return torch.cat(tau, 1), torch.cat(fr, 1)


def _by_level(s, fn, ng):
    """fn on the lower and the upper points of the layer quantities s; two [nlay][n][ng] arrays."""
    nlay, n = s["pav"].shape
    lo = s["low"].reshape(-1)
    a = torch.empty(nlay * n, ng, dtype=torch.float64, device=lo.device)
    b = torch.empty_like(a)
    for m, low in ((lo, True), (~lo, False)):
        sub = {k: v.reshape(-1)[m] for k, v in s.items()}
        a[m], b[m] = fn(sub, low)
    return a.view(nlay, n, ng), b.view(nlay, n, ng)


def _lw_cloud(cols, T, direct, cpathfac):
    """Cloud optical depth [nlay][n][16] (cldprop) and the fractions [nlay][n]."""
    cl = _surface_first(cols, "clouds", 1)
    cf = cl[0]
    if direct:
        tc = cl[1][..., None].expand(*cf.shape, 16)
    else:
        raw = cols["clouds"].flip(1)
        liq, ice = (raw[1] * cpathfac).to(torch.float64), (raw[3] * cpathfac).to(torch.float64)
        fac = cl[2] - 1.5
        i = _trunc(fac).clamp(1, 57)
        A = T["lw_absliq1"].t()
        tl = (liq[..., None] * (A[i - 1] + (fac - i)[..., None] * (A[i] - A[i - 1]))).clamp(min=0.0)
        ia = T["lw_absice1"][_trunc(T["lw_ipat"]) - 1]
        ti = (ice[..., None] * (ia[:, 0] + ia[:, 1] / cl[4].clamp(13.0, 130.0)[..., None])).clamp(min=0.0)
        snow = torch.where((cl[7] > 0) & (cl[8] > 10), 1.5 * f32(1.05756) * cl[7] / cl[8].clamp(min=1.0),
                           torch.zeros_like(cf))
        tc = torch.where(liq[..., None] > 0, tl, 0.0) + torch.where(ice[..., None] > 0, ti, 0.0) + \
            (f32(0.33e-3) * cl[5] + snow)[..., None]
    on = (cf > 0) & (cf > f32(1e-6)).any(0)[None]
    return torch.where(on[..., None], tc, torch.zeros_like(tc)), cf


def _overlap(cf):
    """rtrnmr's overlap factors, upward sweep: fractions cf[1..nlay] met in order 1, 2, ... (cf[0] the value
    below the first, cf[nlay + 1] above the last).  Returns lst [nlay + 2] and the six factors [nlay + 2]."""
    nl = cf.shape[0] - 2
    eps = f32(1e-6)
    z = torch.zeros_like(cf[0])
    F = {k: [z] * (nl + 2) for k in ("clr1", "clr2", "cld1", "cld2", "cmb1", "cmb2")}
    lst = [torch.zeros_like(z, dtype=torch.bool)] * (nl + 2)
    lst[1] = cf[1] > eps
    r1, r2 = z, z
    W = torch.where
    for k in range(1, nl):
        a, c0, cm = cf[k + 1], cf[k], cf[k - 1]
        lst[k + 1] = (a > eps) & (c0 <= eps)
        on, up, st = c0 > eps, a >= c0, lst[k]
        fmx, fmn = torch.maximum(c0, cm), torch.minimum(c0, cm)
        # growing cover
        g2 = W(st, W(c0 < 1, (a - c0) / (1 - c0), z), W(a > fmx, (a - fmx) / (1 - fmx), z))
        g1 = W(st, z, W(a < fmx, (a - c0) / (cm - c0), r2))
        # shrinking cover
        s2 = W(st, (c0 - a) / c0, W(a <= fmn, (fmn - a) / fmn, z))
        s1 = W(st, z, W(a <= fmn, r1, (c0 - a) / (c0 - fmn)))
        F["clr1"][k + 1], F["clr2"][k + 1] = W(on & up, g1, z), W(on & up, g2, z)
        F["cld1"][k + 1], F["cld2"][k + 1] = W(on & ~up, s1, z), W(on & ~up, s2, z)
        F["clr2"][k] = W(on & st, z, F["clr2"][k])
        F["cld2"][k] = W(on & st, z, F["cld2"][k])
        hit = W(up, (F["clr1"][k + 1] > 0) | (F["clr2"][k + 1] > 0), (F["cld1"][k + 1] > 0) | (F["cld2"][k + 1] > 0))
        one = torch.ones_like(z)
        r1, r2 = W(on, W(hit & up, one, z), r1), W(on, W(hit & ~up, one, z), r2)
        F["cmb1"][k + 1] = W(on, F["clr1"][k + 1] * F["cld2"][k] * cm, z)
        F["cmb2"][k + 1] = W(on, F["cld1"][k + 1] * F["clr2"][k] * (1 - cm), z)
    return lst, F


def _mt_masks(cols, ngpt, seed0, lw):
    """McICA sub-column words [words][nlay][n] (maximum-random overlap) and bits [nlay][n][ngpt]: MT19937 seeded
    by column, one draw per (g-point, layer), the single-precision recursion of the generator."""
    cf = cols["clouds"][0].flip(0)
    nlay, n = cf.shape
    if lw:
        cf = torch.where((cf > 1.0e-6).any(0)[None], cf, torch.zeros_like(cf))
    else:
        cf = torch.where(cf < 1.0e-12, torch.zeros_like(cf), cf)
    M32 = 0xFFFFFFFF
    seed = seed0 + 1 + cols["_first"] + torch.arange(n, device=cf.device)
    pw = [1]
    for _ in range(623):
        pw.append(pw[-1] * 69069 & M32)
    mt = (seed[:, None] * torch.tensor(pw, device=cf.device)[None]) & M32

    def mix(hi, lo, far):
        y = (hi & 0x80000000) | (lo & 0x7FFFFFFF)
        return far ^ (y >> 1) ^ ((y & 1) * 0x9908B0DF)

    out = []
    for _ in range(-(-ngpt * nlay // 624)):
        a = mt[:, :227]
        mt = mt.clone()
        mt[:, :227] = mix(a, mt[:, 1:228], mt[:, 397:624])
        for b0 in (227, 454):
            b1 = min(b0 + 227, 623)
            mt[:, b0:b1] = mix(mt[:, b0:b1], mt[:, b0 + 1:b1 + 1], mt[:, b0 - 227:b1 - 227])
        mt[:, 623] = mix(mt[:, 623], mt[:, 0], mt[:, 396])
        y = mt ^ (mt >> 11)
        y = y ^ ((y << 7) & 0x9D2C5680)
        y = y ^ ((y << 15) & 0xEFC60000)
        y = y ^ (y >> 18)
        ys = torch.where(y >= 2 ** 31, y - 2 ** 32, y).to(torch.int32).to(torch.float32)
        out.append(torch.where(ys < 0, ys + 4294967296.0, ys) / 4294967296.0)
    rnd = torch.cat(out, 1)[:, :ngpt * nlay].view(n, ngpt, nlay)
    bits = torch.empty(nlay, n, ngpt, dtype=torch.bool, device=cf.device)
    prev = None
    for k in range(nlay):
        cd = rnd[:, :, k]
        if k:
            tem = (1.0 - cf[k - 1])[:, None]
            cd = torch.where(prev > tem, prev, cd * tem)
        prev = cd
        bits[k] = cd >= (1.0 - cf[k])[:, None]
    nw = (ngpt + 31) // 32
    pad = torch.zeros(nlay, n, nw * 32, dtype=torch.int64, device=cf.device)
    pad[..., :ngpt] = bits
    words = (pad.view(nlay, n, nw, 32) << torch.arange(32, device=cf.device)).sum(-1)
    words = torch.where(words >= 2 ** 31, words - 2 ** 32, words).to(torch.int32)
    return words.permute(2, 0, 1).contiguous(), bits


def _lw_exact(cols, case, cpathfac=1.5):
    T = _tables()
    ex, tfn, tautb, _ = _luts()
    s = _lw_points(cols, T)
    nlay, n = s["pav"].shape
    taug, fracs = _by_level(s, lambda p, low: _lw_gas(p, T, low), 140)
    dv = taug.device
    band = torch.tensor([b for b in range(16) for _ in range(LW_NS[b + 1] - LW_NS[b])], device=dv)
    if "faerlw" in cols:
        f = _surface_first(cols, "faerlw", 2)
        taug = taug + (f[0] * (1.0 - f[1])).permute(1, 2, 0)[..., band]
    # Planck functions at the levels 0..nlay (0: the surface) and of the layers
    tz = _surface_first(cols, "tlvl")
    tl = torch.cat([cols["tsfg"].to(torch.float64)[None], s["tav"]])

    def planck(t):
        i = _trunc(t - 159.0).clamp(1, 180)
        tot = T["lw_totplnk"].t()
        return T["lw_delwave"] * (tot[i - 1] + (t - torch.trunc(t))[..., None] * (tot[i] - tot[i - 1]))

    pklay, pklev = planck(tl), planck(tz)
    # diffusivity from the column water
    t1, t2 = (s["dry"] + s["c0"]).sum(0), s["c0"].sum(0)
    pw = 10.0 * t2 / ((28.9644 / 18.0154) * t1 * 9.80665) * _surface_first(cols, "plvl")[0]
    A0 = (1.66, 1.55, 1.58, 1.66, 1.54, 1.454, 1.89, 1.33, 1.668) + (1.66,) * 7
    A1 = (0.0, 0.25, 0.22, 0.0, 0.13, 0.446, -0.10, 0.40, -0.006) + (0.0,) * 7
    A2 = (0.0, -12.0, -11.7, 0.0, -0.72, -0.243, 0.19, -0.062, 0.414) + (0.0,) * 7
    sec = torch.stack([torch.full_like(pw, f32(1.66)) if b in (0, 3, 9) else
                       (f32(A0[b]) + f32(A1[b]) * torch.exp(f32(A2[b]) * pw)).clamp(f32(1.5), f32(1.8))
                       for b in range(16)], -1)[:, band]
    em = cols["sfcemis"].to(torch.float64)
    em = torch.where((em > f32(1e-6)) & (em <= 1), em, torch.ones_like(em))[:, None]
    tcld, cf = _lw_cloud(cols, T, case["clouds"] == "direct", cpathfac)
    mc = case["route"] == "mcica"
    out = {}
    if mc:
        words, bits = _mt_masks(cols, 140, 140, True)
        out["lw_mask"] = words
    rnd = case["iovrlw"] == 0
    one, zero = torch.ones(1, n, dtype=torch.float64, device=dv), torch.zeros(1, n, dtype=torch.float64, device=dv)
    lstu, Fu = _overlap(torch.cat([one, cf, zero]))
    lstd, Fd = _overlap(torch.cat([zero, cf.flip(0), one]))
    eps, c06, bp = f32(1e-6), f32(0.06), 1.0 / f32(0.278)

    def terms(k):
        od = (sec * taug[k]).clamp(min=0.0)
        thin = od <= c06
        it = _trunc(10000.0 * (od / (bp + od)) + 0.5)
        at = torch.where(thin, od - 0.5 * od * od, 1.0 - ex[it])
        gf = torch.where(thin, f32(0.166667) * od, tfn[it])
        od = torch.where(thin, od, tautb[it])
        bl = pklay[k + 1][:, band]
        du, dd = pklev[k + 1][:, band] - bl, pklev[k][:, band] - bl
        pf = fracs[k]
        g = {"at": at, "gd": pf * (bl + dd * gf) * at, "gu": pf * (bl + du * gf) * at}
        oc = sec * tcld[k][:, band]
        ot = od + oc
        thin = ot < c06
        it = _trunc(10000.0 * (ot / (bp + ot)) + 0.5)
        a = torch.where(thin, ot - 0.5 * ot * ot, 1.0 - ex[it])
        tf = torch.where(thin, f32(0.166667) * ot, tfn[it])
        g.update(a=a, td=pf * (bl + dd * tf) * a, tu=pf * (bl + du * tf) * a, oc=oc)
        return g

    def sweep(order, lst, F, up, tot, clr):
        """One pass; lst / F are met in sweep order.  Returns the radiance changes and the final state."""
        inc, incc, levels = {}, {}, []
        tt = cc = rr = torch.zeros_like(tot)
        for step, k in enumerate(order):
            g = terms(k)
            src, ts = (g["gu"], g["tu"]) if up else (g["gd"], g["td"])
            trn, clf = 1.0 - g["at"], cf[k][:, None]
            incc[k] = src - clr * g["at"]
            if mc or rnd:
                cl = bits[k] if mc else (clf >= eps).expand_as(tot)
                fr = torch.ones_like(clf) if mc else clf
                ef = 1.0 - (1.0 - torch.exp(-g["oc"])) * fr
                S = src + fr * (ts - src)
                cab = -torch.expm1(-g["oc"]) * fr
                inc[k] = torch.where(cl, S - tot * (g["at"] + cab - g["at"] * cab), src - tot * g["at"])
                tot = torch.where(cl, tot * trn * ef + S, tot * trn + src)
            else:
                st = lst[step + 1][:, None]
                tt = torch.where(st, clf * tot, tt)
                cc = torch.where(st, tot - clf * tot, cc)
                rr = torch.where(st, torch.zeros_like(rr), rr)
                cl = clf >= eps
                trt = 1.0 - g["a"]
                f = {q: v[step + 2][:, None] for q, v in F.items()}
                t2 = tt * trt + clf * ts
                c2 = cc * trn + (1.0 - clf) * src
                inc[k] = torch.where(cl, clf * ts + (1.0 - clf) * src - (tt * g["a"] + cc * g["at"]),
                                     src - tot * g["at"])
                tot = torch.where(cl, t2 + c2, tot * trn + src)
                rm = rr * (f["clr1"] * trn + f["cld1"] * trt) - f["cmb1"] * src + f["cmb2"] * ts
                r2 = -rm + f["clr2"] * (c2 + rm) - f["cld2"] * (t2 - rm)
                tt, cc, rr = torch.where(cl, t2 + r2, tt), torch.where(cl, c2 - r2, cc), torch.where(cl, r2, rr)
            clr = clr * trn + src
            levels.append((tot.sum(-1), clr.sum(-1)))
        return inc, incc, levels, tot, clr

    F2 = {"up": Fu, "dn": Fd}
    z = torch.zeros(n, 140, dtype=torch.float64, device=dv)
    # the factors used at layer k are those stored at the level the sweep enters next: k + 1 upward (step + 2)
    pad = {q: {k: v + [torch.zeros_like(v[0])] for k, v in f.items()} for q, f in F2.items()}
    dinc, dincc, dlev, dt, dc = sweep(range(nlay - 1, -1, -1), lstd, pad["dn"], False, z, z)
    rad0 = em * fracs[0] * pklay[0][:, band]
    ut, uc = rad0 + (1.0 - em) * dt, rad0 + (1.0 - em) * dc
    uinc, uincc, ulev, tt, tc = sweep(range(nlay), lstu, pad["up"], True, ut, uc)
    flx = 0.5 * math.pi * 2.0e4
    hf = 9.80665 * 1.0e-2 / 1.0046e3

    def heat(a, b):
        return torch.stack([-(a[k] + b[k]) * flx * (hf / s["dlp"][k]) for k in range(nlay - 1, -1, -1)])

    tot = lambda d: [d[k].sum(-1) for k in range(nlay)]                          # noqa: E731
    out["htlw"] = heat(tot(dinc), tot(uinc))
    out["topflw"] = torch.stack([tt.sum(-1), tc.sum(-1)]) * flx
    out["sfcflw"] = torch.stack([ut.sum(-1), uc.sum(-1), dt.sum(-1), dc.sum(-1)]) * flx
    if case["profiles"]:
        out["hlw0"] = heat(tot(dincc), tot(uincc))
        out["hlwb"] = torch.stack([heat([dinc[k][:, a:b].sum(-1) for k in range(nlay)],
                                        [uinc[k][:, a:b].sum(-1) for k in range(nlay)])
                                   for a, b in zip(LW_NS[:-1], LW_NS[1:])])
        zz = torch.zeros_like(tt.sum(-1))
        up = [(ut.sum(-1), uc.sum(-1))] + ulev                  # levels 0..nlay, surface first
        dn = dlev[::-1] + [(zz, zz)]
        out["lwflxprf"] = torch.stack([torch.stack([v[i] for v in lv[::-1]])
                                       for lv, i in ((up, 0), (dn, 0), (up, 1), (dn, 1))]) * flx
    return out


# --- shortwave
def _sw_points(cols, T):
    plf, p, t = (_surface_first(cols, k) for k in ("plvl", "plyr", "tlyr"))
    q, o = _surface_first(cols, "qlyr"), _surface_first(cols, "olyr")
    gas = _surface_first(cols, "gasvmr", 1)
    dl = plf[:-1] - plf[1:]
    h = (q * (f32(28.9644) / f32(18.0154)) / (1.0 - q)).clamp(min=0.0)
    o3 = (o * (f32(28.9644) / f32(47.9982))).clamp(min=0.0)
    tem0 = (1.0 - h) * f32(28.9644) + h * f32(18.0154)
    cd = f32(1.0e-20) * f32(1.0e3) * f32(6.0221415e23) * dl / (f32(100.0) * f32(9.80665) * tem0 * (1.0 + h))
    tc = f32(1.0e-12) * cd
    s = {"pav": p, "dl": dl, "c1": (cd * h).clamp(min=0.0), "c2": torch.maximum(tc, cd * gas[0]),
         "c3": (cd * o3).clamp(min=0.0), "c4": torch.maximum(tc, cd * gas[1]), "c5": torch.maximum(tc, cd * gas[2]),
         "c6": torch.maximum(tc, cd * gas[3])}
    s["cm"] = cd + s["c1"]
    forf = p * (f32(296.0) / f32(1013.0)) / (t * (1.0 + h))
    plog = torch.log(p)
    jp = _trunc(36.0 - 5.0 * (plog + f32(0.04))).clamp(1, 58)
    fp = 5.0 * (T["sw_preflog"][jp - 1] - plog)
    t1, t2 = (t - T["sw_tref"][jp - 1]) / 15.0, (t - T["sw_tref"][jp]) / 15.0
    jt, jt1 = _trunc(3.0 + t1).clamp(1, 4), _trunc(3.0 + t2).clamp(1, 4)
    ft, ft1 = t1 - (jt - 3), t2 - (jt1 - 3)
    s.update(jp=jp, jt=jt, jt1=jt1, f10=(1.0 - fp) * ft, f00=(1.0 - fp) * (1.0 - ft), f11=fp * ft1,
             f01=fp * (1.0 - ft1))
    lo = plog > f32(4.56)
    a, b, c = (332.0 - t) / 36.0, (t - 188.0) / 36.0, (t - 188.0) / f32(7.2)
    i, j = _trunc(a).clamp(1, 2), (_trunc(c) - 7).clamp(1, 9)
    z = torch.zeros_like(c)
    s["if"], s["ff"] = torch.where(lo, i, torch.full_like(i, 3)), torch.where(lo, a - i, b - 1.0)
    s["is"], s["fs"] = torch.where(lo, j, torch.ones_like(j)), torch.where(lo, c - (j + 7), z)
    s["sfac"], s["ffac"] = torch.where(lo, h * forf, z), forf
    nlay = p.shape[0]
    k = torch.arange(1, nlay + 1, device=p.device)[:, None]
    lt = torch.where(lo, k, torch.zeros_like(k)).amax(0)
    s["lt"] = torch.where(lt == 0, torch.full_like(lt, nlay), lt)
    return s


def _sw_gas(s, T, k8, kw):
    """Gas and Rayleigh optical depths [nlay][n][112]."""
    nlay, n = s["pav"].shape
    dv = s["pav"].device
    q = {k: v.reshape(-1) for k, v in s.items() if k != "lt"}
    k = torch.arange(1, nlay + 1, device=dv)[:, None].expand(nlay, n).reshape(-1)
    lt, k8, kw = (v[None].expand(nlay, n).reshape(-1) for v in (s["lt"], k8, kw))
    nspa = (9, 9, 9, 9, 1, 9, 9, 1, 9, 1, 0, 1, 9, 1)
    nspb = (1, 5, 1, 1, 1, 5, 1, 0, 1, 0, 0, 1, 5, 1)
    low = k <= lt
    ia = ((q["jp"] - 1) * 5 + (q["jt"] - 1), q["jp"] * 5 + (q["jt1"] - 1))
    ib = ((q["jp"] - 13) * 5 + (q["jt"] - 1), (q["jp"] - 12) * 5 + (q["jt1"] - 1))
    om, swom = 1.0 - f32(1e-6), f32(0.999999)
    taug = torch.zeros(nlay * n, 112, dtype=torch.float64, device=dv)
    taur = torch.zeros_like(taug)

    for bi in range(14):
        jb = bi + 16
        sl = slice(SW_NS[bi], SW_NS[bi + 1])
        tb = lambda key: T[f"sw{jb}_{key}"]                                       # noqa: E731,B023
        id0 = torch.where(low, ia[0] * nspa[bi], ib[0] * nspb[bi])
        id1 = torch.where(low, ia[1] * nspa[bi], ib[1] * nspb[bi])

        def pick(m):
            p = {key: v[m] for key, v in q.items()}
            p["id0"], p["id1"] = id0[m], id1[m]                                    # noqa: B023
            return p

        def sum4(p, A):
            out = 0.0
            for i, fa, fb in ((p["id0"], p["f00"], p["f10"]), (p["id1"], p["f01"], p["f11"])):
                i1 = (i + 1).clamp(1, A.shape[0])
                out = out + fa[:, None] * _rows(A, i1) + fb[:, None] * _rows(A, (i1 + 1).clamp(max=A.shape[0]))
            return out

        def sum8(p, A, x1, strr, x2, mult, cap, o1):
            sc = x1 + strr * x2
            sm = mult * torch.where(sc > 0, x1 / sc, torch.zeros_like(sc)).clamp(max=cap)
            j = _trunc(sm)
            fs = sm - j
            out, M = 0.0, A.shape[0]
            for i, fa, fb in ((p["id0"], p["f00"], p["f10"]), (p["id1"], p["f01"], p["f11"])):
                i1 = (i + 1 + j).clamp(1, M)
                for f, off in (((1 - fs) * fa, 0), (fs * fa, 1), ((1 - fs) * fb, o1), (fs * fb, o1 + 1)):
                    out = out + f[:, None] * _rows(A, (i1 + off).clamp(max=M))
            return sc[:, None] * out, j, fs

        def SF(p):
            return p["sfac"][:, None] * _lerp(tb("selfref"), p["is"], p["fs"])     # noqa: B023

        def FF(p):
            return p["ffac"][:, None] * _lerp(tb("forref"), p["if"], p["ff"])      # noqa: B023

        def put(m, v):
            taug[m, sl] = v                                                        # noqa: B023

        ray = {17: 6.86e-10, 19: 2.29e-09, 21: 9.41e-09, 22: 1.54e-08, 29: 9.30e-11}.get(jb)
        if ray is not None:
            taur[:, sl] = (q["cm"] * f32(ray))[:, None]
        elif jb != 24:
            taur[:, sl] = q["cm"][:, None] * tb("rayl")
        if jb in (16, 18, 19):
            p = pick(low)
            x2, strr, cap = {16: (p["c5"], tb("strrat") if jb == 16 else 0, om),
                             18: (p["c5"], T["sw_strrat"][2], swom), 19: (p["c2"], f32(5.49281e+0), swom)}[jb]
            put(low, sum8(p, tb("absa"), p["c1"], strr, x2, 8.0, cap, 9)[0] + p["c1"][:, None] * (SF(p) + FF(p)))
            m = {16: k >= lt, 18: ~low, 19: (k >= lt) & (k >= k8 + 1)}[jb]
            p = pick(m)
            put(m, (p["c2"] if jb == 19 else p["c5"])[:, None] * sum4(p, tb("absb")))
        elif jb in (17, 21):
            strr = T["sw_strrat"][1] if jb == 17 else f32(4.53210e-03)
            m = low if jb == 17 else k < lt
            p = pick(m)
            put(m, sum8(p, tb("absa"), p["c1"], strr, p["c2"], 8.0, om, 9)[0] + p["c1"][:, None] * (SF(p) + FF(p)))
            p = pick(~m)
            put(~m, sum8(p, tb("absb"), p["c1"], strr, p["c2"], 4.0, om, 5)[0] + p["c1"][:, None] * FF(p))
        elif jb == 20:
            for m, key in ((low, "absa"), (~low, "absb")):
                p = pick(m)
                g = sum4(p, tb(key)) + FF(p)
                put(m, p["c1"][:, None] * (g + SF(p) if key == "absa" else g) + p["c5"][:, None] * tb("absch4"))
        elif jb == 22:
            o2c = f32(4.35e-4) / (f32(350.0) * 2.0)
            p = pick(low)
            put(low, sum8(p, tb("absa"), p["c1"], f32(3.63328e-02), p["c6"], 8.0, om, 9)[0] +
                p["c1"][:, None] * (SF(p) + FF(p)) + (o2c * p["c6"])[:, None])
            p = pick(~low)
            put(~low, (p["c6"] * f32(1.6))[:, None] * sum4(p, tb("absb")) + (o2c * p["c6"])[:, None])
        elif jb == 23:
            m = low & ~((k >= k8 + 1) & (k >= lt))
            p = pick(m)
            put(m, p["c1"][:, None] * (f32(1.029) * sum4(p, tb("absa")) + SF(p) + FF(p)))
        elif jb == 24:
            p = pick(low)
            g, j, fs = sum8(p, tb("absa"), p["c1"], f32(1.24692e-1), p["c6"], 8.0, swom, 9)
            put(low, g + p["c3"][:, None] * tb("abso3a") + p["c1"][:, None] * (SF(p) + FF(p)))
            R = tb("rayla")
            taur[low, sl] = p["cm"][:, None] * (R[j] + fs[:, None] * (R[j + 1] - R[j]))
            p = pick(~low)
            put(~low, p["c6"][:, None] * sum4(p, tb("absb")) + p["c3"][:, None] * tb("abso3b"))
            taur[~low, sl] = p["cm"][:, None] * tb("raylb")
        elif jb == 25:
            p = pick(low)
            put(low, p["c1"][:, None] * sum4(p, tb("absa")) + p["c3"][:, None] * tb("abso3a"))
            m = (k >= kw + 1) & (k >= lt)
            put(m, q["c3"][m][:, None] * tb("abso3b"))
        elif jb == 27:
            for m, key in ((k < lt, "absa"), (k >= lt, "absb")):
                p = pick(m)
                put(m, p["c3"][:, None] * sum4(p, tb(key)))
        elif jb == 28:
            p = pick(low)
            put(low, sum8(p, tb("absa"), p["c3"], tb("strrat"), p["c6"], 8.0, swom, 9)[0])
            m = (k >= kw + 1) & (k >= lt)
            p = pick(m)
            put(m, sum8(p, tb("absb"), p["c3"], tb("strrat"), p["c6"], 4.0, swom, 5)[0])
        elif jb == 29:
            p = pick(low)
            put(low, p["c1"][:, None] * (sum4(p, tb("absa")) + SF(p) + FF(p)) + p["c2"][:, None] * tb("absco2"))
            p = pick(~low)
            put(~low, p["c2"][:, None] * sum4(p, tb("absb")) + p["c1"][:, None] * tb("absh2o"))
    return taug.view(nlay, n, 112), taur.view(nlay, n, 112)


def _sw_source(s, T):
    """Solar source of the g-points, [n][112]."""
    nlay, n = s["pav"].shape
    dv, lt, jp = s["pav"].device, s["lt"], s["jp"]
    out = torch.empty(n, 112, dtype=torch.float64, device=dv)
    kk = torch.arange(1, nlay, device=dv)[:, None]
    for b in range(14):
        jb, sl, ng = b + 16, slice(SW_NS[b], SW_NS[b + 1]), SW_NS[b + 1] - SW_NS[b]
        ibd = int(T["sw_ibx"][b])
        if jb in (16, 20, 23, 25, 26, 27, 29):
            v = T["sw_sfluxref01"].reshape(-1, 16)[ibd - 1, :ng]
            out[:, sl] = v * T["sw_scalekur"][0] if jb == 27 else v
            continue
        two = jb in (17, 28)
        lr = int(T["sw_layreffr"][b])
        hit = (jp[:-1] < lr) & (jp[1:] >= lr) & ((kk >= lt) if two else (kk <= lt - 1))
        first = torch.where(hit, kk, torch.full_like(kk, 10 ** 6)).amin(0)
        ks = torch.where(first < 10 ** 6, first + 1, torch.full_like(first, nlay) if two else lt)
        at = lambda i: s[f"c{i}"].gather(0, (ks - 1)[None])[0]                     # noqa: E731,B023
        c1, c2 = at(int(T["sw_ix1"][b])), at(int(T["sw_ix2"][b]))
        sm = T["sw_specwt"][b] * (c1 / (c1 + T["sw_strrat"][b] * c2)).clamp(max=f32(0.999999))
        j = _trunc(sm)
        R = (T["sw_sfluxref02"] if two else T["sw_sfluxref03"])[ibd - 1]
        out[:, sl] = R[j, :ng] + (sm - j)[:, None] * (R[j + 1, :ng] - R[j, :ng])
    return out


def _sw_cloud(cols, T, direct):
    cl = _surface_first(cols, "clouds", 1)
    cf = cl[0]
    if direct:
        t = cl[1][..., None].expand(*cf.shape, 14)
        sc = t * cl[2][..., None]
        res = (t, sc, sc * cl[3][..., None])
    else:
        def opt(pre, path, fac, top):
            i = _trunc(fac).clamp(1, top)
            f = (fac - i)[..., None]
            v = []
            for key in ("ext", "ssa", "asy"):
                A = T[f"sw_{key}{pre}"].t()
                x = (A[i - 1] + f * (A[i] - A[i - 1])).clamp(min=0.0)
                v.append(x if key == "ext" else x.clamp(max=1.0))
            on = (path > 0)[..., None]
            tau = torch.where(on, path[..., None] * v[0], 0.0)
            return tau, tau * v[1], tau * v[1] * v[2]
        liq = opt("liq1", cl[1], cl[2] - 1.5, 57)
        ice = opt("ice3", cl[3], ((f32(1.0315) * cl[4]).clamp(5.0, 140.0) - 2.0) / 3.0, 45)
        # the workloads carry no rain or snow (clouds 5 and 7 are zero), whose terms vanish with their paths
        res = tuple(a + b for a, b in zip(liq, ice))
    on = (cf > f32(1e-12))[..., None]
    return [torch.where(on, v, torch.zeros_like(v)) for v in res], cf


def _sw_exact(cols, case, day):
    """The solve of the sunlit columns; day = (laytrop minimum of the 8-column group, of the chunk)."""
    T = _tables()
    extb = _luts()[3]
    s = _sw_points(cols, T)
    nlay, n = s["pav"].shape
    taug, taur = _sw_gas(s, T, *day)
    dv = taug.device
    band = torch.tensor([b for b in range(14) for _ in range(SW_NS[b + 1] - SW_NS[b])], device=dv)
    cz = cols["coszen"].to(torch.float64)[:, None]
    snt = 1.0 / cz
    ssol = (f32(SOLCON) / f32(1368.22)) * cz
    zsol = ssol * _sw_source(s, T)
    (ctau, cssa, casy), cf = _sw_cloud(cols, T, case["clouds"] == "direct")
    ftiny, om = f32(1e-12), 1.0 - f32(1e-6)
    z0, z1 = torch.ones_like(cf[0]), torch.ones_like(cf[0])
    for k in range(nlay):                                   # maximum-random clear-sky view fraction
        on, gap = cf[k] > ftiny, z1 < 1
        z0 = torch.where(~on & gap, z0 * z1, z0)
        z1 = torch.where(on, torch.minimum(z1, 1.0 - cf[k]), torch.ones_like(z1))
    z0 = z0 * z1
    z0 = torch.where(z0 <= ftiny, torch.zeros_like(z0), torch.where(z0 > om, torch.ones_like(z0), z0))
    z1 = 1.0 - z0
    mc = case["route"] == "mcica"
    out = {}
    if mc:
        bits = cols["_sw_bits"]
    cloudy = z1 > (0.0 if mc else f32(1e-6))
    lcf = torch.where(z1 > 0, cf / z1.clamp(min=1e-300), torch.zeros_like(cf))
    ae = None
    if "faersw" in cols:
        f = _surface_first(cols, "faersw", 2).permute(0, 2, 3, 1)
        ae = (f[0], f[0] * f[1], f[2] * f[1] * f[0])
    mode = case["iswmode"]

    def expm(zb):
        it = _trunc((zb / (1.0 / f32(0.278) + zb)) * 10000.0 + 0.5).clamp(0, 10000)
        return torch.where(zb <= f32(0.06), 1.0 - zb + 0.5 * zb * zb, extb[it])

    def layer(t0, s0, y0):
        w = (s0 / t0).clamp(max=om)
        a = y0 / s0.clamp(min=ftiny)
        a2 = w * a * a
        t1, w1 = (1.0 - a2) * t0, (w - a2) / (1.0 - a2)
        y1 = a / (1.0 + a)
        y3 = 0.75 * y1
        if mode == 2:
            g1, g2, g3 = 2.0 - w1 * (1.25 + y3), 0.75 * w1 * (1.0 - y1), 0.5 - y3 * cz
        else:
            r3 = f32(1.7320508)
            g1, g2, g3 = r3 * (2.0 - w1 * (1.0 + y1)) * 0.5, r3 * w1 * (1.0 - y1) * 0.5, (1.0 - r3 * y1 * cz) * 0.5
        g4 = 1.0 - g3
        A1, A2 = g1 * g4 + g2 * g3, g1 * g3 + g2 * g4
        kk = torch.sqrt((g1 - g2) * (g1 + g2))
        rp = kk * cz
        pp = 1.0 - rp * rp
        e8 = f32(1e-8)
        pp = torch.where(pp.abs() < e8, torch.where(pp < 0, -e8, e8), pp)
        r4, r5 = pp * (kk + g1), pp * (kk - g1)
        e1, e2 = expm((kk * t1).clamp(max=500.0)), expm((t1 * snt).clamp(max=500.0))
        x1, x2 = 1.0 / e1, 1.0 / e2
        D = r4 * x1 + r5 * e1
        bad = D.abs() <= e8
        dn = w1 / torch.where(bad, torch.ones_like(D), D)
        rb = (((1 - rp) * (A2 + kk * g3) * x1 - (1 + rp) * (A2 - kk * g3) * e1 - 2 * kk * (g3 - A2 * cz) * e2) * dn)
        tb = e2 * (1.0 - ((1 + rp) * (A1 + kk * g4) * x1 - (1 - rp) * (A1 - kk * g4) * e1 -
                          2 * kk * (g4 + A1 * cz) * x2) * dn)
        rb = torch.where(bad, torch.full_like(D, e8), rb.clamp(0.0, 1.0))
        tb = torch.where(bad, e2, tb.clamp(0.0, 1.0))
        dd = r4 / (D * (kk + g1))
        return [rb, (g2 * (x1 - e1) * dd).clamp(0.0, 1.0), tb, (2 * kk * dd).clamp(0.0, 1.0), expm(t1 * snt),
                expm(t0 * snt)]

    ibd = torch.tensor([1, 1, 1, 1, 1, 1, 1, 1, 0, 2, 2, 2, 2, 1], device=dv)[band]
    alb = cols["sfcalb"].to(torch.float64)

    def surface(a, b):
        return torch.where(ibd == 1, a[:, None], torch.where(ibd == 2, b[:, None], (0.5 * (a + b))[:, None]))

    ab, ad = surface(alb[0], alb[2]), surface(alb[1], alb[3])
    passes = []
    clear = []
    for k in range(nlay):
        a = [x[k][:, band] for x in ae] if ae else (0.0, 0.0, 0.0)
        t0 = (taur[k] + taug[k] + a[0]).clamp(min=ftiny)
        s0 = taur[k] + a[1]
        y0 = a[2] + torch.zeros_like(s0)
        clear.append((t0, s0, y0, layer(t0, s0, y0)))
    for ps in range(2):
        R = []
        for k in range(nlay):
            t0, s0, y0, c = clear[k]
            if ps:
                o = layer(t0 + ctau[k][:, band], s0 + cssa[k][:, band], y0 + casy[k][:, band])
                zc = lcf[k][:, None]
                on = (zc > ftiny) & cloudy[:, None]
                if mc:
                    c = [torch.where(on & bits[k], y, x) for x, y in zip(c, o)]
                else:
                    c = [torch.where(on, (1.0 - zc) * x + zc * y, x) for x, y in zip(c, o)]
            R.append(c)
        ub, ud = [ab], [ad]
        for k in range(nlay):
            rb, rd, tb, td, e3, _ = R[k]
            den = 1.0 / (1.0 - ud[k] * rd)
            ub.append(rb + (td * ((tb - e3) * ud[k] + e3 * ub[k])) * den)
            ud.append(rd + td * td * ud[k] * den)
        tdn, rdn, tdb = torch.ones_like(ab), torch.zeros_like(ab), torch.ones_like(ab)
        fu, fd = [None] * (nlay + 1), [None] * (nlay + 1)
        dir0 = torch.ones_like(ab)
        for k in range(nlay, -1, -1):
            den = 1.0 / (1.0 - rdn * ud[k])
            fu[k] = zsol * (tdb * ub[k] + (tdn - tdb) * ud[k]) * den
            fd[k] = zsol * (tdb + (tdn - tdb + tdb * ub[k] * rdn) * den)
            if k:
                rb, rd, tb, td, e3, e4 = R[k - 1]
                den = 1.0 / (1.0 - rd * rdn)
                tdn, rdn, tdb = (tdb * tb + (td * ((tdn - tdb) + tdb * rb * rdn)) * den, rd + td * td * rdn * den,
                                 e3 * tdb)
                dir0 = dir0 * e4
        passes.append((fu, fd, zsol * dir0))
    w0 = torch.where(cloudy, torch.zeros_like(z0) if mc else z0, torch.ones_like(z0))
    w1 = torch.where(cloudy, torch.ones_like(z0) if mc else z1, torch.zeros_like(z0))
    t0 = torch.where(cloudy, z0, torch.ones_like(z0)) if not mc else w0
    t1 = torch.where(cloudy, z1, torch.zeros_like(z0)) if not mc else w1

    def tot(i, k):                                          # band and g-point sums are left to the caller
        return t0[:, None] * passes[0][i][k] + t1[:, None] * passes[1][i][k]

    net = [w0[:, None] * (passes[0][1][k] - passes[0][0][k]) + w1[:, None] * (passes[1][1][k] - passes[1][0][k])
           for k in range(nlay + 1)]
    rdl = (9.80665 * 1.0e-2 / 1.0046e3) / s["dl"]

    def heat(lv):
        return torch.stack([(lv[k + 1] - lv[k]) * rdl[k] for k in range(nlay - 1, -1, -1)])

    out["htsw"] = heat([v.sum(-1) for v in net])
    cu, cd = passes[0][0], passes[0][1]
    S = lambda x: x.sum(-1)                                                        # noqa: E731
    out["topfsw"] = torch.stack([S(tot(0, nlay)), S(cd[nlay]), S(cu[nlay])])
    out["sfcfsw"] = torch.stack([S(tot(0, 0)), S(tot(1, 0)), S(cu[0]), S(cd[0])])
    uv = band == 11
    beam = t0[:, None] * passes[0][2] + t1[:, None] * passes[1][2]
    diff = tot(1, 0) - beam
    nir, vis = torch.where(ibd == 1, 1.0, torch.where(ibd == 0, 0.5, 0.0)), \
        torch.where(ibd == 2, 1.0, torch.where(ibd == 0, 0.5, 0.0))
    out["fdncmp"] = torch.stack([S(cd[0] * uv), S(tot(1, 0) * uv), S(beam * nir), S(diff * nir), S(beam * vis),
                                 S(diff * vis)])
    if case["profiles"]:
        out["hsw0"] = heat([S(cd[k] - cu[k]) for k in range(nlay + 1)])
        out["htswb"] = torch.stack([heat([v[:, a:b].sum(-1) for v in net]) for a, b in zip(SW_NS[:-1], SW_NS[1:])])
        lv = range(nlay, -1, -1)
        out["swflxprf"] = torch.stack([torch.stack([S(tot(0, k)) for k in lv]), torch.stack([S(tot(1, k)) for k in lv]),
                                       torch.stack([S(cu[k]) for k in lv]), torch.stack([S(cd[k]) for k in lv])])
    return out


def _exact_request(cols, case):
    n = int(cols["tsfg"].shape[0])
    T = _tables()
    parts, res = case["parts"], {}

    def piece(idx, first):
        d = {k: v[..., idx].contiguous() for k, v in cols.items()}
        d["_first"] = first
        return d

    def write(key, idx, v):
        if key not in res:
            res[key] = torch.zeros(*v.shape[:-1], n, dtype=v.dtype, device=v.device)
        res[key][..., idx] = v

    if parts != "sw":
        for c0 in range(0, n, EXACT_CHUNK):
            idx = slice(c0, min(n, c0 + EXACT_CHUNK))
            for k, v in _lw_exact(piece(idx, c0), case).items():
                write(k, idx, v)
    if parts != "lw":
        bits = []
        if case["route"] == "mcica":
            for c0 in range(0, n, EXACT_CHUNK):
                idx = slice(c0, min(n, c0 + EXACT_CHUNK))
                words, b = _mt_masks(piece(idx, c0), 112, 1, False)
                write("sw_mask", idx, words)
                bits.append(b)
            bits = torch.cat(bits, 1)
        day = torch.nonzero(cols["coszen"] >= 1.0e-4)[:, 0]
        nd = day.numel()
        lts = []
        for c0 in range(0, nd, EXACT_CHUNK):
            lts.append(_sw_points(piece(day[c0:c0 + EXACT_CHUNK], 0), T)["lt"])
        if nd:
            lt = torch.cat(lts)

            def groups(size):
                pad = -nd % size
                g = torch.cat([lt, torch.full((pad,), 10 ** 6, device=lt.device, dtype=lt.dtype)]).view(-1, size)
                return g.amin(1).repeat_interleave(size)[:nd]

            k8, kw = groups(8), groups(32768)
            for c0 in range(0, nd, EXACT_CHUNK):
                sel = slice(c0, min(nd, c0 + EXACT_CHUNK))
                d = piece(day[sel], 0)
                if len(bits):
                    d["_sw_bits"] = bits[:, day[sel]]
                for k, v in _sw_exact(d, case, (k8[sel], kw[sel])).items():
                    write(k, day[sel], v)
        else:
            nl = case["nlay"]
            for key, shape in (("htsw", (nl,)), ("topfsw", (3,)), ("sfcfsw", (4,)), ("fdncmp", (6,))):
                res[key] = torch.zeros(*shape, n, dtype=torch.float64, device=cols["tsfg"].device)
            if case["profiles"]:
                for key, shape in (("hsw0", (nl,)), ("htswb", (14, nl)), ("swflxprf", (4, nl + 1))):
                    res[key] = torch.zeros(*shape, n, dtype=torch.float64, device=cols["tsfg"].device)
    return res


def exact(case, seed):
    # The whole radiation call's front end is defined by single-precision statements (cloud-type and terminator
    # decisions), so it has no 64-bit counterpart to compare with.
    if case["kind"] == "call" or sum(_sizes(case)) > EXACT_COLUMNS:
        return None
    res = [_exact_request(_columns(n, seed + 1000003 * r, case), case) for r, n in enumerate(_sizes(case))]
    return res[0] if len(res) == 1 else res
