"""Performance cases: the work a program built on umwm_gb300 has the library do.

A wave case ("kind": "wave") is one forecast interval through the umwm_top
entry points: the host program hands over an analysis (set_state), runs the
model over one dtg (umwm_run: the dynamic time steps, then the Stokes drift and
the diagnostics) and reads the results back.  Every case is one of the forms in
which the library is used: small and large domains, regular and longitude-
latitude grids, land, currents, moving winds, sea ice, other spectral grids,
ensembles, the host-driven, graph-driven and autotuned loops, and the
ocean-coupled step that keeps the source terms and reads two-dimensional
fields only.  A network case ("kind": "forward" or "grad") is a batch through
the source-term surrogate: inference, or the loss and its gradient.

The seed of a case's input draws the analysis spectrum, its swell and the
friction velocity (a batch and its targets for the network); the grid, the
forcing and the network's weights belong to the case.

exact() restates the model in float64 (the reference's formulas, with the
spectrum cut at zero after the propagation as umwm_gpu.h documents).
"""
import math

import numpy as np
import torch

import umwm_gb300 as U
from umwm_gb300.configs import holland_wind, sea_mask_from_z, smooth_field
from umwm_gb300.namelist import DEFAULTS, make_namelist

START = "2012-01-01 00:00:00"
FPAD, HID, NFEAT, NBIN = 1344, 512, 1341, 1332  # the surrogate's padded width, hidden width, inputs, outputs

# two-dimensional fields a program reads after an interval
FIELDS = ("ht", "mwp", "mss", "momx", "momy", "cgmxx", "cgmyy", "ustar", "taux", "tauy", "taux_form")
# what a program reads of each ensemble member
MEMBER = ("ht", "mwp", "ustar", "taux", "tauy")
# what an ocean model takes from the wave model each coupling interval
OCEAN = ("ht", "mwp", "ustar", "taux", "tauy", "us", "vs", "taux_ocntop", "tauy_ocntop", "taux_ocnbot", "tauy_ocnbot",
         "taux_snl", "tauy_snl", "epsx_ocn", "epsy_ocn", "epsx_atm", "epsy_atm", "tailocnx", "tailocny", "taux1",
         "tauy1", "taux2", "tauy2", "taux3", "tauy3")

WAVE = {"kind": "wave", "grid": "flat", "dx": 2000.0, "om": 37, "pm": 36, "dtg": 1800, "loop": "host", "ice": False,
        "ocean": False, "members": 1, "spectrum": True, "stokes": False, "grid_seed": 1}


def _names(c):
    """Fields the program reads; "stokes": the Stokes drift profile too."""
    if c["ocean"]:
        return OCEAN
    return (MEMBER if c["members"] > 1 else FIELDS) + (("us", "vs") if c["stokes"] else ())


def _wave(**kw):
    return dict(WAVE, **kw)


def listed():
    return [
        # the shipped namelist's grid (21x11, 10 km, constant wind, dtg 1 h): a pond or a test deployment
        _wave(name="pond_21x11", mm=21, nm=11, dx=10000.0, dtg=3600, stokes=True),
        # a bay with a ragged coast and currents, on a coarser spectral grid
        _wave(name="bay_61x47", mm=61, nm=47, grid="land", om=30, pm=24, grid_seed=2),
        # the idealised fetch-limited basin of the repository's workloads (100x100 at 5 km), graph-driven loop
        _wave(name="fetch_100x100", mm=100, nm=100, dx=5000.0, dtg=3600, loop="graph", stokes=True),
        # a skewed longitude-latitude grid (curvilinear propagation) with land and currents
        _wave(name="lonlat_121x90", mm=121, nm=90, grid="lonlat", grid_seed=3),
        # a marginal ice zone: ice fraction from 0 to 0.9 across the domain
        _wave(name="ice_150x113", mm=150, nm=113, grid="land", ice=True, grid_seed=4),
        # a wave model coupled to an ocean model every 10 minutes: stress('ocn'), no spectrum to the host
        _wave(name="coupled_200x160", mm=200, nm=160, grid="land", dtg=600, ocean=True, spectrum=False, loop="graph",
              grid_seed=5),
        # a regional forecast hour, host-driven loop
        _wave(name="region_301x287", mm=301, nm=287, grid="land", dtg=3600, grid_seed=6),
        # a moving hurricane over a shelf, autotuned and graph-driven, as a production run starts
        _wave(name="hurricane_400x360", mm=400, nm=360, grid="hurricane", loop="tuned", grid_seed=7),
        # the largest domain: a forecast hour of a basin, gridded results only
        _wave(name="basin_640x600", mm=640, nm=600, grid="land", dtg=3600, loop="graph", spectrum=False, grid_seed=8),
        # an ensemble of small hurricanes advanced as one model, each member's gridded results
        _wave(name="ensemble_8", mm=80, nm=60, grid="hurricane", members=8, loop="graph", spectrum=False,
              grid_seed=9),
        # the surrogate's inference on a domain's worth of input rows, and one training batch's loss and gradient
        {"name": "net_forward_12000", "kind": "forward", "rows": 12000},
        {"name": "net_grad_8192", "kind": "grad", "rows": 8192},
    ]


def draw(rng):
    kind = rng.choices(["wave", "forward", "grad"], [10, 1, 1])[0]
    if kind != "wave":
        n = int(math.exp(rng.uniform(math.log(64), math.log(12000))))
        return {"kind": kind, "rows": max(64, n // 64 * 64) if kind == "grad" else n}
    grid = rng.choice(["flat", "land", "land", "lonlat", "hurricane"])
    members = rng.choice([1, 1, 1, 1, 3, 6]) if grid == "hurricane" else 1
    cells = math.exp(rng.uniform(math.log(200), math.log(250000))) / members
    cells = max(cells, 400 if grid != "flat" else 200)
    aspect = math.exp(rng.uniform(-0.7, 0.7))
    mm, nm = max(11, int(math.sqrt(cells * aspect))), max(11, int(math.sqrt(cells / aspect)))
    om, pm = rng.choice([(37, 36), (37, 36), (37, 36), (30, 24), (25, 32), (37, 48), (33, 16)])
    ocean = members == 1 and rng.random() < 0.15
    return _wave(mm=mm, nm=nm, grid=grid, dx=rng.choice([2000.0, 3000.0, 5000.0, 10000.0]), om=om, pm=pm,
                 dtg=rng.choice([600, 900, 1800]), loop=rng.choice(["host", "graph", "graph"]),
                 ice=grid == "land" and rng.random() < 0.25, ocean=ocean, spectrum=not ocean, members=members,
                 stokes=rng.random() < 0.3,
                 grid_seed=rng.randrange(1000))


# ---- the case's domain: grid, forcing, namelist --------------------------------------------------------------

def _domain(c, member=0):
    """Grid, depth and forcing of one member as host arrays; a function of the case alone."""
    mm, nm, dx = c["mm"] + 7 * member, c["nm"] + 5 * member, c["dx"]
    rng = np.random.Generator(np.random.Philox(1000 * c["grid_seed"] + member))
    d = {"mm": mm, "nm": nm, "dx": dx, "z": None, "lon": None, "lat": None, "forcing": None}
    x = (np.arange(mm) * dx)[:, None] * np.ones((1, nm))
    y = (np.arange(nm) * dx)[None, :] * np.ones((mm, 1))
    if c["grid"] in ("land", "lonlat"):
        s = dx / 2000.0

        def smooth(cells):
            return smooth_field((mm, nm), max(2.0, cells / s), rng)

        land, dep, u, v, cu, cv = (smooth(k) for k in (25, 25, 100, 100, 25, 25))
        depth = np.clip(np.exp(np.log(300.0) + 1.3 * dep), 10.0, 5000.0)
        z = np.where(land < np.quantile(land, 0.2), 5.0, -depth).astype(np.float32)
        z[1, 1] = -50.0  # at least one wet point
        w, q = 20.0 / np.hypot(u, v).max(), 1.0 / np.hypot(cu, cv).max()
        f = [{"uw": (u * w * g).astype(np.float32), "vw": (v * w * g).astype(np.float32),
              "uc": (cu * q).astype(np.float32), "vc": (cv * q).astype(np.float32)} for g in (1.0, 1.05)]
        if c["ice"]:
            ice = np.clip(1.3 * x / x.max() - 0.2 + 0.1 * dep, 0.0, 0.9).astype(np.float32)
            for snap in f:
                snap["fice"] = ice
        d.update(z=z, forcing=f)
        if c["grid"] == "lonlat":
            m, n, step = np.arange(mm)[:, None], np.arange(nm)[None, :], dx / 1.112e5
            d["lon"] = (-80.0 + step * m + 0.04 * step * n).astype(np.float32)
            d["lat"] = (20.0 + step * n + 0.02 * step * m).astype(np.float32)
    elif c["grid"] == "hurricane":
        depth = 20.0 + 2980.0 * np.minimum(x / 300e3, 1.0)
        depth = depth * (1 + 0.05 * np.clip(smooth_field((mm, nm), 5.0, rng) / 3.0, -1, 1))
        head, cur = rng.uniform(0, 2 * np.pi, size=2)
        f = []
        for t in (0.0, float(c["dtg"])):
            xc, yc = 0.5 * mm * dx + 5.0 * t * np.cos(head), 0.5 * nm * dx + 5.0 * t * np.sin(head)
            uw, vw = holland_wind(x, y, xc, yc, heading=head)
            f.append({"uw": uw, "vw": vw, "uc": np.full((mm, nm), 0.5 * np.cos(cur), np.float32),
                      "vc": np.full((mm, nm), 0.5 * np.sin(cur), np.float32)})
        d.update(z=(-depth).astype(np.float32), forcing=f)
    z = d["z"] if d["z"] is not None else np.full((mm, nm), -1000.0, np.float32)
    d["mask"] = sea_mask_from_z(z)
    d["wet"] = np.nonzero(d["mask"])  # row-major over (m, n): the library's order of wet points
    forced = d["forcing"] is not None
    sec = c["dtg"]
    d["stop"] = "2012-01-01 %02d:%02d:%02d" % (sec // 3600, sec // 60 % 60, sec % 60)
    wm, wn = d["wet"]
    half = len(wm) // 2
    d["nml"] = make_namelist(mm=mm, nm=nm, om=c["om"], pm=c["pm"], delx=dx, dely=dx, dpt=1000.0, dtg=sec,
                             topoFromFile=d["z"] is not None, gridFromFile=d["lon"] is not None, winds=forced,
                             currents=forced, seaice=bool(c["ice"]), restart=False, startTimeStr=START,
                             stopTimeStr=d["stop"], xpl=int(wm[half]) + 1, ypl=int(wn[half]) + 1)
    return d


def _stage(d):
    for var, key in (("z", "z"), ("lon", "lon"), ("lat", "lat")):
        if d[key] is not None:
            U.put_gridtopo(var, d[key])
    if d["forcing"] is not None:
        for t, snap in zip((START, d["stop"]), d["forcing"]):
            for var, fld in snap.items():
                U.put_forcing(t, var, fld)


# ---- dispersion and the analysis spectrum --------------------------------------------------------------------

def _spectral(om, pm, dev):
    fmin, fmax = DEFAULTS["fmin"], DEFAULTS["fmax"]
    dlnf = (math.log(fmax) - math.log(fmin)) / (om - 1)
    f = torch.exp(math.log(fmin) + torch.arange(om, dtype=torch.float64, device=dev) * dlnf)
    dth = 2 * math.pi / pm
    th = (torch.arange(1, pm + 1, dtype=torch.float64, device=dev) - 0.5 * (pm + 1)) * dth
    return f, th, dlnf, dth


def _dispersion(f, d, dlnf):
    """k, phase and group speed, wavenumber step over (points, frequencies): Newton steps with surface
    tension until a step in k d is below 1e-2, as the reference iterates."""
    g, sfct, rhow0 = DEFAULTS["g"], DEFAULTS["sfct"], float(DEFAULTS["rhow0"])
    d = d[:, None]
    fn = 2 * math.pi * torch.sqrt(d / g) * f
    b = sfct / (rhow0 * g * d * d)
    k, going = fn * fn, torch.ones_like(fn, dtype=torch.bool)
    for _ in range(1000):
        t = torch.tanh(k)
        dk = -(fn * fn - k * t * (1 + b * k * k)) / (3 * b * k * k * t + t + k * (1 + b * k * k) * (1 - t * t))
        k = torch.where(going, k - dk, k)
        going = going & (dk.abs() > 1e-2)
        if not bool(going.any()):
            break
    k = k.abs() / d
    kd = torch.clamp(k * d, max=20.0)
    cp = 2 * math.pi * f / k
    cg = cp * (0.5 + k * d / torch.sinh(2 * kd) + sfct * k * k / (rhow0 * g + sfct * k * k))
    return k, kd, cp, cg, 2 * math.pi * dlnf * f / cg.abs()


def _depth(d, dev):
    wm, wn = d["wet"]
    z = np.full((d["mm"], d["nm"]), -1000.0, np.float32) if d["z"] is None else d["z"]
    return torch.tensor(np.maximum(np.abs(z[wm, wn].astype(np.float64)), DEFAULTS["dmin"]), device=dev)


def _wind(d, snap, dev):
    wm, wn = d["wet"]
    if d["forcing"] is None:
        n = len(wm)
        return (torch.full((n,), float(DEFAULTS["wspd0"]), dtype=torch.float64, device=dev),
                torch.zeros(n, dtype=torch.float64, device=dev))
    s = d["forcing"][snap]
    return (torch.tensor(s["uw"][wm, wn].astype(np.float64), device=dev),
            torch.tensor(s["vw"][wm, wn].astype(np.float64), device=dev))


def _pinned(t):
    """The tensor as a host array in pinned memory, where a program keeps what it hands over repeatedly."""
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t).numpy()


def _analysis(c, d, seed):
    """Spectrum F(im, pm, om) and ustar(im) as float32 host arrays: a wind sea in the local wind (JONSWAP,
    broad spreading) and a swell of random direction, each bin perturbed, drawn from the seed."""
    dev = "cuda"
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    f, th, dlnf, dth = _spectral(c["om"], c["pm"], dev)
    u, v = _wind(d, 0, dev)
    u, v = (torch.full_like(u, float(DEFAULTS["wspd0"])), torch.zeros_like(v)) if d["forcing"] is None else (u, v)
    w = torch.clamp(torch.hypot(u, v), min=1.0)[:, None]
    wd = torch.atan2(v, u)[:, None]
    fp = torch.clamp(1.8 * 0.13 * DEFAULTS["g"] / w, 0.08, 0.5)
    hs = torch.clamp(0.012 * w * w, 0.05, 6.0)
    r = torch.rand(4, generator=gen, device=dev, dtype=torch.float64)

    def shape(fp_, gamma):
        sig = torch.where(f <= fp_, 0.07, 0.09)
        s = f ** -5 * torch.exp(-1.25 * (fp_ / f) ** 4) * gamma ** torch.exp(-((f - fp_) ** 2) / (2 * sig ** 2 * fp_ ** 2))
        s = s * f * dlnf
        return s / s.sum(1, keepdim=True)

    def spread(ang, s):
        q = torch.cos(0.5 * (th - ang)).abs() ** (2 * s)
        return q / (q.sum(1, keepdim=True) * dth)

    swell = 0.4 + 0.6 * r[0]
    k, _, _, _, dwn = _dispersion(f, _depth(d, dev), dlnf)
    wind = ((hs / 4) ** 2 * shape(fp, 3.3) / (k * dwn))[:, None, :] * spread(wd, 4.0)[:, :, None]
    sw = ((swell / 4) ** 2 * shape(0.07 + 0.04 * r[1] + 0 * w, 5.0) / (k * dwn))[:, None, :]
    sw = sw * spread(2 * math.pi * r[2] + 0 * w, 12.0)[:, :, None]
    noise = 0.8 + 0.4 * torch.rand(wind.shape, generator=gen, device=dev, dtype=torch.float32)
    F = ((wind + sw) * noise).float()
    us = torch.sqrt(torch.where(w > 11, (0.49 + 0.065 * w) * 1e-3, torch.full_like(w, 1.2e-3))) * w
    us = (us[:, 0] * (0.95 + 0.1 * r[3])).float()
    return _pinned(F), _pinned(us)


def _weights():
    """The network's weights (a trained network's scale), the same for every seed."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(77)

    def normal(rows, cols, s):
        return torch.randn(rows, cols, generator=gen, device="cuda") * s

    w1, w2, w3 = normal(HID, FPAD, math.sqrt(2.0 / NFEAT)), normal(HID, HID, math.sqrt(2.0 / HID)), normal(FPAD, HID, HID ** -0.5)
    w1[:, NFEAT:] = 0
    w3[NBIN:] = 0
    b = [normal(1, n, 0.05)[0] for n in (HID, HID, FPAD)]
    b[2][NBIN:] = 0
    return w1, b[0], w2, b[1], w3, b[2]


def _batch(c, seed):
    """Input rows in the range of the log-spectrum features and, for the gradient, targets."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    X = torch.zeros(c["rows"], FPAD, device="cuda")
    X[:, :NFEAT] = torch.randn(c["rows"], NFEAT, generator=gen, device="cuda")
    T = torch.zeros(c["rows"], FPAD, device="cuda")
    T[:, :NBIN] = 0.3 * torch.randn(c["rows"], NBIN, generator=gen, device="cuda")
    return X, T


# ---- prepare, run, work ---------------------------------------------------------------------------------------

def prepare(case, seed):
    c = dict(case)
    if c["kind"] != "wave":
        U.surrogate_init(37, 36, seed=1)
        U.surrogate_set_params(torch.cat([w.reshape(-1) for w in _weights()]).cpu().numpy())
        X, T = _batch(c, seed)
        return {"c": c, "X": _pinned(X), "T": _pinned(T)}
    doms = [_domain(c, m) for m in range(c["members"])]
    states = [_analysis(c, d, 1000003 * int(seed) + m) for m, d in enumerate(doms)]
    torch.cuda.empty_cache()
    U.clear_inputs()
    for d in doms:
        _stage(d)
        if c["members"] > 1:
            U.ensemble_add(d["nml"])
    if c["members"] > 1:
        U.ensemble_initialize()
    else:
        U.umwm_initialize(nml_text=doms[0]["nml"])
    U.set_option("use_graph", 0 if c["loop"] == "host" else 1)
    if c["ocean"]:
        U.set_option("stress_ocn", 1)
    s = {"c": c, "stop": doms[0]["stop"], "states": states}
    if c["loop"] == "tuned":  # the tuner measures its candidates on the first intervals of a run
        U.set_option("autotune", 1)
        U.set_state(*states[0])
        for _ in range(3):
            U.umwm_run(START, s["stop"])
    return s


def run(s):
    c = s["c"]
    if c["kind"] == "forward":
        return U.surrogate_forward(s["X"])
    if c["kind"] == "grad":
        loss, g = U.surrogate_grad(s["X"], s["T"])
        return {"loss": np.float32(loss), "grad": g}
    many = len(s["states"]) > 1
    for m, st in enumerate(s["states"]):
        if many:
            U.select_member(m)
        U.set_state(*st)
    U.umwm_run(START, s["stop"])
    out = []
    for m in range(len(s["states"])):
        if many:
            U.select_member(m)
        r = {n: U.get_field(n) for n in _names(c)}
        if c["spectrum"]:
            r["F"] = U.get_state()[0]
        out.append(r)
    return out


def work(case):
    """Wave cases: the interval's substeps (the propagation's time step limit divides the interval) each read
    and write the spectrum once in the source step and once in the propagation, the least that the grid-wide
    time step and the neighbours allow; the analysis in, the spectrum and fields out.  Network cases: rows in
    and out, weights (and their gradient)."""
    c = case
    if c["kind"] != "wave":
        n, mul = c["rows"], FPAD * HID + HID * HID + HID * FPAD
        w = 4.0 * (mul + 2 * HID + FPAD)
        if c["kind"] == "forward":
            return {"bytes": 8.0 * n * FPAD + w, "flops": 2.0 * n * mul}
        return {"bytes": 8.0 * n * FPAD + 2 * w, "flops": 2.0 * n * (3 * mul - FPAD * HID)}
    bins = points = 0
    for m in range(c["members"]):
        wet = (c["mm"] + 7 * m - 2) * (c["nm"] + 5 * m - 2) * (0.8 if c["grid"] in ("land", "lonlat") else 1.0)
        bins += wet * c["om"] * c["pm"]
        points += wet
    cgmax = 26.0 if c["grid"] == "flat" else 28.0  # m/s, the lowest frequency in intermediate depth
    cfl = math.cos(0.25 * math.pi - math.pi / c["pm"]) if c["pm"] % 8 == 0 else math.sqrt(0.5)
    steps = math.ceil(c["dtg"] / (0.98 * cfl * c["dx"] / cgmax))
    io = 4.0 * bins * (2 if c["spectrum"] else 1) + 4.0 * points * (14 + (84 if c["stokes"] or c["ocean"] else 0))
    return {"bytes": 16.0 * bins * steps + io, "flops": 60.0 * bins * steps}


# ---- the model in float64 ---------------------------------------------------------------------------------------

def exact(case, seed):
    c = dict(case)
    if c["kind"] != "wave":
        return _exact_net(c, seed)
    w = work(c)
    if w["bytes"] > 1.6e11 or c["loop"] == "tuned":  # over about 20 seconds
        return None
    return [_exact_wave(c, _domain(c, m), 1000003 * int(seed) + m) for m in range(c["members"])]


def _exact_net(c, seed):
    w1, b1, w2, b2, w3, b3 = (t.double() for t in _weights())
    X, T = (t.double() for t in _batch(c, seed))

    def gelu(z):
        return 0.5 * z * (1 + torch.erf(z / math.sqrt(2)))

    def dgelu(z):
        return 0.5 * (1 + torch.erf(z / math.sqrt(2))) + z * torch.exp(-0.5 * z * z) / math.sqrt(2 * math.pi)

    z1 = X @ w1.T + b1
    h1 = gelu(z1)
    z2 = h1 @ w2.T + b2
    h2 = gelu(z2)
    Y = h2 @ w3.T + b3
    if c["kind"] == "forward":
        return Y
    d = Y - T
    d[:, NBIN:] = 0
    n = c["rows"] * NBIN
    dY = 2 * d / n
    dz2 = (dY @ w3) * dgelu(z2)
    dz1 = (dz2 @ w2) * dgelu(z1)
    g = [dz1.T @ X, dz1.sum(0), dz2.T @ h1, dz2.sum(0), dY.T @ h2, dY.sum(0)]
    return {"loss": float((d * d).sum() / n), "grad": torch.cat([t.reshape(-1) for t in g])}


def _spacing(d):
    """dx, dy (m) and the grid's curvature angle over (mm, nm)."""
    mm, nm = d["mm"], d["nm"]
    if d["lon"] is None:
        return np.full((mm, nm), d["dx"]), np.full((mm, nm), d["dx"]), np.zeros((mm, nm))
    lon, lat = np.deg2rad(d["lon"].astype(np.float64)), np.deg2rad(d["lat"].astype(np.float64))

    def dist(lo1, lo2, la1, la2):
        s = np.sin(0.5 * (la2 - la1)) ** 2 + np.cos(la1) * np.cos(la2) * np.sin(0.5 * (lo2 - lo1)) ** 2
        return 6.371009e6 * 2 * np.arcsin(np.sqrt(s))

    dx, dy, cv = np.empty((mm, nm)), np.empty((mm, nm)), np.empty((mm, nm))
    lm, am = 0.5 * (lon[1:] + lon[:-1]), 0.5 * (lat[1:] + lat[:-1])
    dx[1:-1] = dist(lm[:-1], lm[1:], am[:-1], am[1:])
    dx[0], dx[-1] = 2 * dx[1] - dx[2], 2 * dx[-2] - dx[-3]
    ln, an = 0.5 * (lon[:, 1:] + lon[:, :-1]), 0.5 * (lat[:, 1:] + lat[:, :-1])
    dy[:, 1:-1] = dist(ln[:, :-1], ln[:, 1:], an[:, :-1], an[:, 1:])
    dy[:, 0], dy[:, -1] = 2 * dy[:, 1] - dy[:, 2], 2 * dy[:, -2] - dy[:, -3]
    dl = lon[2:] - lon[:-2]
    cv[1:-1] = np.arctan2(np.sin(dl) * np.cos(lat[2:]),
                          np.cos(lat[:-2]) * np.sin(lat[2:]) - np.sin(lat[:-2]) * np.cos(lat[2:]) * np.cos(dl))
    cv[0], cv[-1] = cv[1], cv[-2]
    return dx, dy, cv - 0.5 * math.pi


def _shelter(w):
    x1, x2, x3, y1, y2, y3 = 15.0, 33.0, 60.0, 0.10, 0.09, 0.06
    s1, s2 = (y1 - 0.04) / x1, (y3 - y2) / (x3 - x2)
    c = 0.65 * (s2 - s1) / (x2 - x1)
    b = s1 - 2 * c * x1
    a = y1 - b * x1 - c * x1 * x1
    end = a + b * x2 + c * x2 * x2
    return torch.where(w <= x1, 0.04 + s1 * w,
                       torch.where(w <= x2, a + b * w + c * w * w, end * torch.exp(-(w - x2) / (1.6 * w))))


def _exact_wave(c, d, seed):
    dev, N = "cuda", DEFAULTS
    om, pm, dtg = c["om"], c["pm"], float(c["dtg"])
    g, kappa, z10, nua, nuw = N["g"], N["kappa"], N["z"], N["nu_air"], N["nu_water"]
    f, th, dlnf, dth = _spectral(om, pm, dev)
    F, ust = _analysis(c, d, seed)
    wm, wn = d["wet"]
    im, mm, nm = len(wm), d["mm"], d["nm"]
    e = torch.tensor(F, device=dev).double()
    ustar = torch.tensor(ust, device=dev).double()
    # unrolled grid: neighbours by wet index (im: the ghost point)
    idx = np.full((mm, nm), im)
    idx[wm, wn] = np.arange(im)

    def near(field, a, b):
        return torch.tensor(field[wm + a, wn + b], device=dev)

    ie, iw, inn, iss = (near(idx, a, b) for a, b in ((1, 0), (-1, 0), (0, 1), (0, -1)))
    DX, DY, CV = _spacing(d)
    dx, dy = near(DX, 0, 0), near(DY, 0, 0)
    dxn, dxs, dye, dyw = (0.5 * (near(D, 0, 0) + near(D, a, b)) for D, a, b in ((DX, 0, 1), (DX, 0, -1), (DY, 1, 0), (DY, -1, 0)))
    k, kd, cp0, cg0, dwn = _dispersion(f, _depth(d, dev), dlnf)
    kdk, k3dk, k4, fkovg = k * dwn, k ** 3 * dwn, k ** 4, f * k / g
    coth = 1 / torch.tanh(0.2 * kd)
    sbf = N["sbf_fac"] * k / torch.sinh(2 * kd) + N["sbp_fac"] * k / torch.cosh(kd) ** 2
    sdv = 4 * nuw * k * k
    l2 = torch.clamp(0.5 * cp0 / f, max=20.0)
    log2z = torch.log(l2 / z10)
    b1, b2 = math.exp(-16 * dlnf ** 2), math.exp(-64 * dlnf ** 2)
    b1, b2 = b1 / (b1 + b2), b2 / (b1 + b2)
    snlf = N["snl_fac"]
    w1, w2 = torch.zeros_like(k), torch.zeros_like(k)
    w1[:, :-2] = snlf * b1 * kdk[:, 1:-1] / kdk[:, :-2]
    w2[:, :-2] = snlf * b2 * kdk[:, 2:] / kdk[:, :-2]

    def ghosted(a, ghost):
        return torch.cat([a, ghost[None]])

    cpG, cgG = ghosted(cp0, cp0.min(0).values), ghosted(cg0, cg0.min(0).values)
    mdx = min(DX[d["mask"] == 1].min(), DY[d["mask"] == 1].min())
    cfl = math.cos(0.25 * math.pi - 0.5 * dth) if pm % 8 == 0 else math.sqrt(0.5)
    dtamin = 0.98 * cfl * mdx / float(cg0.max())
    cth, sth = torch.cos(th), torch.sin(th)
    cv = near(CV, 0, 0)[:, None] if d["lon"] is not None else torch.zeros(1, 1, dtype=torch.float64, device=dev)
    cc, sc = torch.cos(th + cv)[:, :, None], torch.sin(th + cv)[:, :, None]
    c2, s2 = torch.cos(2 * th), torch.sin(2 * th)
    cth_, sth_ = cth[:, None], sth[:, None]
    sina, f1, f2 = N["sin_fac"], N["sin_diss1"] / N["sin_fac"], N["sin_diss2"] / N["sin_diss1"]
    sA = 2 * math.pi * N["sds_fac"] * f
    rhoa, rhow = N["rhoa0"], float(N["rhow0"])
    rr = rhoa / rhow
    ks, forced = torch.arange(1, om + 1, device=dev), d["forcing"] is not None
    full = {}
    if forced:
        for var in d["forcing"][0]:
            snaps = [s[var].astype(np.float64) for s in d["forcing"]]
            if var in ("uc", "vc"):
                snaps = [s * (d["mask"] == 1) for s in snaps]
            full[var] = snaps
    surf = [torch.zeros(im, dtype=torch.float64, device=dev)] * 2  # surface Stokes drift of the last interval

    def at(var, a, s, da=0, db=0):
        b, n = full[var]
        return near(b, da, db) * a + near(n, da, db) * s

    zero = torch.zeros(im, dtype=torch.float64, device=dev)
    sumt, first, keep = 0.0, True, None
    while sumt < dtg:
        s = sumt / dtg
        a = 1 - s
        if forced:
            u, v = at("uw", a, s), at("vw", a, s)
            uc, vc = at("uc", a, s), at("vc", a, s)
            cur = {q: (at("uc", a, s, *o), at("vc", a, s, *o)) for q, o in (("e", (1, 0)), ("w", (-1, 0)), ("n", (0, 1)), ("s", (0, -1)))}
        else:
            u, v, uc, vc = zero + float(N["wspd0"]), zero, zero, zero
            cur = {q: (zero, zero) for q in "ewns"}
        fice = at("fice", a, s) if "fice" in full else zero
        wspd, wdir = torch.clamp(torch.hypot(u, v), min=1e-2), torch.atan2(v, u)
        fc = torch.clamp(0.53 * g / wspd, max=N["fprog"])
        oc = torch.clamp((f[None, :om - 2] < fc[:, None]).sum(1), min=1)
        prog = (ks <= oc[:, None])[:, None, :]
        # wind input
        cw = torch.cos(wdir[:, None] - th)[:, :, None]
        U_ = (wspd[:, None] + 2.5 * ustar[:, None] * log2z)[:, None, :]
        x = U_ * cw - cp0[:, None, :] - uc[:, None, None] * cth_ - vc[:, None, None] * sth_
        x = sina * x.abs() * x
        x = torch.where(x > 0, x * _shelter(wspd)[:, None, None] / sina, torch.where(cw > 0, x * f1 * f2, x * f1))
        ssin = ((1 - fice) * 2 * math.pi * rr)[:, None, None] * x * fkovg[:, None, :]
        del x
        ssin = torch.where(prog, ssin, torch.clamp(ssin, min=0.0))
        # dissipation: the mean-square slope of the longer waves, projected on each direction
        m = [torch.einsum("ipo,p->io", e, q) * k3dk * 0.5 * dth for q in (torch.ones_like(th), c2, s2)]
        A, B, C = (torch.cumsum(q, 1) - q for q in m)
        t = (1 + N["mss_fac"] * (A[:, None, :] + B[:, None, :] * c2[:, None] + C[:, None, :] * s2[:, None])) ** 2
        sds = sA * t * (e * k4[:, None, :]) ** N["sds_power"]
        # downshifting
        de = sds * e
        snl = -snlf * de
        snl[:, :, :-2] += w1[:, None, :-2] * de[:, :, 1:-1] + w2[:, None, :-2] * de[:, :, 2:]
        snl = torch.where(prog, snl, 0.0)
        del de
        sds = sds * coth[:, None, :]
        sdt = N["sdt_fac"] * math.sqrt(rr) * ustar[:, None] * k
        hs = 4 * torch.sqrt(torch.einsum("ipo,io->i", e, kdk) * dth)
        sv = torch.where(fice > N["fice_lth"], -5.35e-6 * torch.clamp(hs, max=3.0), 0.0)
        sink = (sbf + sdt + sdv - 2 * cg0 * sv[:, None])[:, None, :]
        arg = torch.where(prog, ssin - sds * (1 - w1 - w2)[:, None, :] - sink, 0.0)
        dts = min(N["explim"] / float(arg.abs().max()), dtamin, dtg - sumt)
        if first:
            dts = 0.0
        sumt += dts
        del arg
        ef = e * torch.exp(dts * (ssin - sds - sink)) + dts * snl
        num = ssin - (sdt + sdv - 2 * cg0 * sv[:, None])[:, None, :]
        eq = torch.clamp(num, min=0.0) / (sA * t * coth[:, None, :])
        ef = torch.where(prog, ef, eq ** (1 / N["sds_power"]) / k4[:, None, :])
        del num, eq, t
        es = torch.cat([0.5 * (e + ef), torch.full((1, pm, om), float(np.finfo(np.float32).tiny), dtype=torch.float64, device=dev)])
        if c["ocean"]:
            keep = (ssin, sds, snl, sdt)
        # propagation
        here = es[:im]
        flux = torch.zeros_like(here)
        any_cur = bool((uc != 0).any() or (vc != 0).any())
        for q, nb, ln, dr, sgn, vel, mine in (("e", ie, dye, cc, 1, 0, uc), ("w", iw, dyw, cc, -1, 0, uc),
                                              ("n", inn, dxn, sc, 1, 1, vc), ("s", iss, dxs, sc, -1, 1, vc)):
            cge = (cg0 + cgG[nb])[:, None, :] * dr
            p, mns = cge + cge.abs(), cge - cge.abs()
            if any_cur:
                uu = (mine + cur[q][vel])[:, None, None]
                p, mns = p + uu + uu.abs(), mns + uu - uu.abs()
            other = es[nb]
            flux += (sgn * ln)[:, None, None] * ((p * here + mns * other) if sgn > 0 else (p * other + mns * here))
            del cge, p, mns, other
        frozen = (fice > N["fice_uth"])[:, None, None]
        ef = torch.where(prog, ef - 0.25 * dts * flux / (dx * dy)[:, None, None], ef)
        # refraction
        rot = 0.5 * (((cpG[ie] - cpG[iw])[:, None, :] * sth_ + (cur["e"][1] - cur["w"][1])[:, None, None]) / dx[:, None, None] -
                     ((cpG[inn] - cpG[iss])[:, None, :] * cth_ + (cur["n"][0] - cur["s"][0])[:, None, None]) / dy[:, None, None])
        rot = torch.where(prog, rot, 0.0)
        fastest = float(rot.max())
        dtr = min(dth / fastest, dts) if fastest > 1.2e-38 else dts
        edge = 0.5 * (rot + torch.roll(rot, -1, 1))
        edge = torch.where(edge > 0, edge * here, edge * torch.roll(here, -1, 1))
        ef = torch.where(prog, ef - dtr * (edge - torch.roll(edge, 1, 1)) / dth, ef)
        ef = torch.where(prog & frozen, 0.0, ef)
        e = torch.clamp(ef, min=0.0)
        del edge, rot, flux, es, here
        # stress: the form drag divides by the phase speed of the previous unrolled point
        prev = torch.cat([cpG[im:], cp0[:-1]])
        es = e * ssin
        tx, ty = (torch.einsum("ipo,p->io", es, q) / prev for q in (cth, sth))
        slope = 0.000112 * wspd ** 2 - 0.01451 * wspd - 1.0186
        kt = k[:, -1] ** slope
        tl = (1e3 ** (slope + 1) - k[:, -1] * kt) / (kt * (slope + 1))
        form = [(q * kdk).sum(1) * rhow * dth * g + q[:, -1] * k[:, -1] * tl * rhow * dth * g for q in (tx, ty)]
        ur, vr = wspd * torch.cos(wdir) - uc - surf[0], wspd * torch.sin(wdir) - vc - surf[1]
        wr, wdr = torch.hypot(ur, vr), torch.atan2(vr, ur)
        cdf = torch.hypot(*form) / (rhoa * wspd ** 2)
        z0 = torch.full_like(wr, 1e-3)
        for _ in range(6):
            usk = kappa * wr / torch.log(z10 / z0)
            z0 = 0.132 * nua / usk
        cds = usk ** 2 / wspd ** 2
        cds = torch.clamp(cds * (1 + 2 * cds / (cds + cdf + 1.2e-38)) / 3, max=1e-2)
        skin = [rhoa * cds * wr ** 2 * torch.cos(wdr), rhoa * cds * wr ** 2 * torch.sin(wdr)]
        tau = [p + q for p, q in zip(form, skin)]
        ustar = torch.sqrt(torch.hypot(*tau) / rhoa)
        first = False
    # Stokes drift and diagnostics of the interval's end
    dep = -torch.tensor(N["depths"], dtype=torch.float64, device=dev)
    depth = _depth(d, dev)
    X, Y = (torch.einsum("ipo,p->io", e, q) for q in (cth, sth))
    us, vs = [], []
    for l in range(len(dep)):
        k_d, arg = k * depth[:, None], 2 * k * (dep[l] + depth[:, None])
        deep = 2 * torch.exp(2 * k * dep[l])
        fin = torch.cosh(torch.clamp(arg, max=50.0)) / torch.sinh(torch.clamp(k_d, max=50.0)) ** 2
        q = 2 * math.pi * f * k * k * torch.where((arg.abs() > 50) | (k_d > 50), deep, fin) * dwn * dth
        q = torch.where((dep[l].abs() > depth)[:, None], 0.0, q)
        us.append((q * X).sum(1))
        vs.append((q * Y).sum(1))
    E = e.sum(1)
    P, icp = (ks <= oc[:, None]).double(), 1 / cp0
    rg = rhow * dth * g
    m0 = (E * kdk).sum(1)
    Ecc, Ess = (torch.einsum("ipo,p->io", e, q * q) for q in (cth, sth))
    out = {"ht": 4 * torch.sqrt(m0 * dth), "mwp": torch.sqrt(m0 / (E * f * f * kdk).sum(1)), "mss": (E * k3dk).sum(1) * dth,
           "momx": (X * kdk * icp * P).sum(1) * rg, "momy": (Y * kdk * icp * P).sum(1) * rg,
           "cgmxx": (Ecc * kdk * icp * cg0 * P).sum(1) * rg, "cgmyy": (Ess * kdk * icp * cg0 * P).sum(1) * rg,
           "ustar": ustar, "taux": tau[0], "tauy": tau[1], "taux_form": form[0], "us": torch.stack(us), "vs": torch.stack(vs)}
    if c["ocean"]:
        out.update(_exact_ocean(e, keep, dict(k=k, kdk=kdk, cp0=cp0, sbf=sbf, sdv=sdv, P=P, cth=cth, sth=sth, b1=b1, b2=b2,
                                              tl=tl, rg=rg, skin=skin, cw=cw)))
    res = {n: out[n] for n in _names(c)}
    if c["spectrum"]:
        res["F"] = e
    return res


def _exact_ocean(e, keep, q):
    """Momentum and energy handed to the ocean, from the spectrum and the last substep's source terms."""
    ssin, sds, snl, sdt = keep
    k, kdk, cp0, icp = q["k"], q["kdk"], q["cp0"], 1 / q["cp0"]
    wm, wl = torch.zeros_like(k), torch.zeros_like(k)
    r1, r2 = cp0[:, 2:] * icp[:, 1:-1], cp0[:, 2:] * icp[:, :-2]
    wm[:, 2:] = q["b1"] * r1 + q["b2"] * r2
    wl[:, 2:] = q["b1"] * (1 - r1) + q["b2"] * (1 - r2)
    out = {}
    for ax, dr in (("x", q["cth"]), ("y", q["sth"])):
        def along(a):
            return torch.einsum("ipo,p->io", a, dr)

        def total(a):
            return (a * kdk).sum(1) * q["rg"]

        E, D, S, W = along(e), along(e * sds), along(snl), along(e * ssin)
        top = (D + E * (sdt + q["sdv"]) - S * wm) * icp
        tail = top[:, -1] * k[:, -1] * q["tl"] * q["rg"]
        out["tailocn" + ax] = tail
        out["tau%s_ocntop" % ax] = total(top) + tail + q["skin"][0 if ax == "x" else 1]
        out["tau%s_ocnbot" % ax] = total(E * q["sbf"] * icp)
        out["tau%s_snl" % ax] = total(S * wl * icp * q["P"])
        out["eps%s_ocn" % ax] = total(D - S * wm)
        out["eps%s_atm" % ax] = total(W)
        for n, sel in (("1", ssin > 0), ("2", (ssin <= 0) & (q["cw"] < 0)), ("3", (ssin <= 0) & (q["cw"] >= 0))):
            out["tau%s%s" % (ax, n)] = total(along(torch.where(sel, e * ssin, 0.0)) * icp)
    return out
