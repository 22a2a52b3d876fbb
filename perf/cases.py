"""The work that programs give this engine, as cases that can be timed and checked.

Every case goes through an entry point that a program calls (`Engine.profile`,
`profile_fit`, `profile_batch`, `batch(...).launch`, `submit` / `wait`, and the
stand-alone fold `ppm_fold_device`), on the tables that the engine keeps
resident: the "wide" lensing tables and the v171019-shaped NSX atmosphere, both
loaded once per process.  A case is a dict of plain values:

  kind        profile | fit | batch | batch_host | served | fold
  atmosphere  nsx | blackbody (profile only; the other kinds are NSX)
  region      point | cap (one disk) | pair (ring + crescent) | prior (random morphologies)
  n_side, bins, nodes (Gauss-Legendre points per bin, 0 = point-sampled phases),
  energies, channels (0 = flux only), interp, precision, fold
  count       profiles of a batch, requests of a served group, flux arrays of a fold

Stars are drawn from the batching prior (mass, radius, spin, inclination,
temperature); the spots of the fixed regions are perturbed as a sampler's
proposals around one geometry are, so that every seed is another input of
about the same size.

`exact` is the same physics in 64 bits, written with torch alone.
"""
import ctypes
import math
import random  # noqa: F401  (draw() takes a random.Random)

import numpy as np
import torch

from gpu_ppm_b200 import _abi, synth
from gpu_ppm_b200.engine import Engine

INTERP = {"4c": 0, "4c_sg": 1, "4c_le": 2, "2l2c_le": 3, "4l": 4}
FOLD = {"bf16x3": 0, "fp32": 1, "fp64": 2}
BEAM = {"iso": 0, "sin2": 1, "cos2": 2}
E_LO, E_HI = 0.2, 12.0  # keV: the range of the spectral grids
U_RANGE, LOGG_RANGE = (0.15, 0.55), (13.7, 14.7)  # the tables' ranges, to which the prior is cut


def listed():
    """Twelve cases over the engine's range, smallest calls first."""
    return [
        # a bolometric-like light curve of a point spot: the smallest call there is, where launches and copies count
        dict(name="lightcurve_point", kind="profile", atmosphere="blackbody", region="point", n_side=256, bins=128,
             nodes=0, energies=1, channels=0, precision="fp64", beaming="iso"),
        # a light curve of a spot of 1 rad (the os1 stars): many rings, one energy
        dict(name="lightcurve_cap", kind="profile", atmosphere="blackbody", region="cap", radius=1.0, n_side=256,
             bins=128, nodes=0, energies=1, channels=0, precision="fp64", beaming="cos2"),
        # blackbody spectrum per phase bin in 64 bits: one disk, N_side 64, 64 energies
        dict(name="spectrum_blackbody", kind="profile", atmosphere="blackbody", region="cap", radius=0.25, n_side=64,
             bins=32, nodes=2, energies=64, channels=0, precision="fp64", beaming="iso"),
        # the smallest size of the served mix, called by itself: a coarse likelihood evaluation
        dict(name="nsx_coarse", kind="profile", atmosphere="nsx", region="cap", radius=0.3, n_side=64, bins=32, nodes=2,
             energies=128, channels=300, interp="2l2c_le", fold="bf16x3"),
        # the two-spot workload, N_side 256, 64 bins, 300 energies and channels: one ordinary profile
        dict(name="nsx_pair", kind="profile", atmosphere="nsx", region="pair", n_side=256, bins=64, nodes=2,
             energies=300, channels=300, interp="2l2c_le", fold="bf16x3"),
        # the precision workload: N_side 512, 128 bins, 1500 channels, folded in 64 bits
        dict(name="nsx_fine_fold64", kind="profile", atmosphere="nsx", region="pair", n_side=512, bins=128, nodes=2,
             energies=300, channels=1500, interp="2l2c_le", fold="fp64"),
        # ragged sizes, cubic in all four axes, three nodes per bin, 32-bit fold
        dict(name="nsx_odd_cubic", kind="profile", atmosphere="nsx", region="pair", n_side=101, bins=45, nodes=3,
             energies=211, channels=157, interp="4c", fold="fp32"),
        # one likelihood evaluation of a sampler: scalars come back
        dict(name="fit_proposal", kind="fit", region="cap", radius=0.2, n_side=128, bins=64, nodes=2, energies=300,
             channels=300, interp="2l2c_le", fold="bf16x3"),
        # a group of mixed requests through the server, as several walkers send them
        dict(name="served_mix", kind="served", count=24, region="prior", n_side=512, bins=128, nodes=2, energies=300,
             channels=1500, interp="2l2c_le", fold="bf16x3"),
        # a host call on mixed profiles: parameters in, flux and counts out
        dict(name="batch_host", kind="batch_host", count=24, region="prior", n_side=256, bins=64, nodes=2, energies=300,
             channels=300, interp="2l2c_le", fold="bf16x3"),
        # the device-resident batch of the benchmark's prior, an eighth of its length
        dict(name="batch_resident", kind="batch", count=512, region="prior", n_side=256, bins=64, nodes=2, energies=300,
             channels=300, interp="2l2c_le", fold="bf16x3"),
        # the response fold of a batch of spectra that are on the device already
        dict(name="fold_tensor", kind="fold", count=1024, bins=64, energies=300, channels=300, fold="bf16x3"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: sizes over their logarithm, odd ones among them."""
    largest = max(_cost(c) for c in listed())
    while True:
        c = _draw_once(rng)
        if _cost(c) <= largest:
            return c


def _draw_once(rng):
    kind = rng.choice(["lightcurve", "spectrum", "profile", "profile", "fit", "served", "batch_host", "batch", "fold"])
    if kind == "lightcurve":
        region = rng.choice(["point", "cap", "cap"])
        c = dict(kind="profile", atmosphere="blackbody", region=region, n_side=_log_int(rng, 48, 512),
                 bins=_log_int(rng, 32, 256), nodes=rng.choice([0, 0, 2]), energies=rng.choice([1, 1, 1, 3]), channels=0,
                 precision=rng.choice(["fp64", "fp64", "fp32"]), beaming=rng.choice(["iso", "sin2", "cos2"]))
        if region == "cap":
            c["radius"] = round(math.exp(rng.uniform(math.log(0.1), 0.0)), 3)
        return c
    if kind == "spectrum":
        return dict(kind="profile", atmosphere="blackbody", region=rng.choice(["cap", "pair"]),
                    radius=round(math.exp(rng.uniform(math.log(0.05), 0.0)), 3), n_side=_log_int(rng, 24, 192),
                    bins=_log_int(rng, 16, 96), nodes=rng.choice([1, 2, 3]), energies=_log_int(rng, 16, 300),
                    channels=0, precision=rng.choice(["fp64", "fp64", "fp32"]), beaming="iso")
    if kind == "fold":
        return dict(kind="fold", count=_log_int(rng, 1, 1024), bins=_log_int(rng, 16, 128),
                    energies=_log_int(rng, 32, 400), channels=_log_int(rng, 24, 1500),
                    fold=rng.choice(["bf16x3", "fp32", "fp64"]))
    nsx = dict(bins=_log_int(rng, 16, 128), nodes=rng.choice([1, 2, 2, 3]), energies=_log_int(rng, 32, 400),
               channels=_log_int(rng, 24, 1500), interp=rng.choice(["2l2c_le", "2l2c_le", "4c", "4c_sg", "4c_le", "4l"]),
               fold=rng.choice(["bf16x3", "bf16x3", "fp32", "fp64"]))
    if kind in ("profile", "fit"):
        region = rng.choice(["cap", "pair", "pair"])
        c = dict(kind=kind, region=region, n_side=_log_int(rng, 32, 512), **nsx)
        if kind == "profile":
            c["atmosphere"] = "nsx"
        if region == "cap":
            c["radius"] = round(math.exp(rng.uniform(math.log(0.02), 0.0)), 3)
        return c
    if kind == "served":
        return dict(kind="served", count=rng.randint(1, 30), region="prior", n_side=rng.choice([128, 256, 512]), **nsx)
    if kind == "batch_host":
        return dict(kind="batch_host", count=_log_int(rng, 2, 24), region="prior", n_side=_log_int(rng, 32, 256), **nsx)
    return dict(kind="batch", count=_log_int(rng, 8, 512), region="prior", n_side=_log_int(rng, 32, 300), **nsx)


# ------------------------------------------------------------------ what a program keeps: the engine and its tables
_KEPT = {}


def _tables():
    if "tables" not in _KEPT:
        _KEPT["tables"] = (synth.lensing("wide"), synth.nsx("v171019", seed=0))
    return _KEPT["tables"]


def _engine():
    if "engine" not in _KEPT:
        lens, nsx = _tables()
        eng = Engine(device=0)
        eng.load_lensing(lens)
        eng.load_nsx(nsx)
        _KEPT["engine"] = eng
    return _KEPT["engine"]


def _energies(n):
    return synth.energy_grid(n, E_LO, E_HI) if n > 4 else np.linspace(1.0, 1.0 + 0.5 * (n - 1), n)


def _response(n_e, n_ch):
    key = ("response", n_e, n_ch)
    if key not in _KEPT:
        _KEPT[key] = synth.response(n_ch, 1000 if n_ch <= 300 else 2 * n_ch, _energies(n_e), seed=0)
    return _KEPT[key]


def _ids(n_e, n_ch):
    """The engine's ids of an energy grid and of a response on it."""
    eng = _engine()
    if ("grid", n_e) not in _KEPT:
        _KEPT["grid", n_e] = eng.add_energy_grid(_energies(n_e))
    g = _KEPT["grid", n_e]
    if not n_ch:
        return g, -1
    if ("rsp", n_e, n_ch) not in _KEPT:
        _KEPT["rsp", n_e, n_ch] = eng.add_response(g, _response(n_e, n_ch))
    return g, _KEPT["rsp", n_e, n_ch]


# ------------------------------------------------------------------ inputs
def _star(rng):
    while True:
        m, r, nu = rng.uniform(1.0, 2.2), rng.uniform(9.0, 15.0), rng.uniform(100.0, 700.0)
        (u0, g0), (u1, g1) = synth.star_u_logg(m, r, nu)
        if U_RANGE[0] <= min(u0, u1) and max(u0, u1) <= U_RANGE[1] and \
                LOGG_RANGE[0] <= min(g0, g1) and max(g0, g1) <= LOGG_RANGE[1]:
            return dict(mass_msun=m, r_eq_km=r, spin_hz=nu, inclination_rad=rng.uniform(30.0, 80.0) * synth.DEG)


def _spots(rng, region, radius, log_t, kt):
    def near(v, rel):
        return v * (1.0 + rel * rng.uniform(-1.0, 1.0))

    warm = dict(logT=log_t, kT_keV=kt)
    if region == "point":
        return [synth.spot(near(60 * synth.DEG, 0.3), 0.0, 0.01, kind=_abi.SPOT_POINT, **warm)]
    if region == "cap":
        return [synth.spot(near(70 * synth.DEG, 0.1), near(0.3, 1.0), near(radius, 0.02), **warm)]
    if region == "pair":
        t1, t2 = near(30 * synth.DEG, 0.05), near(120 * synth.DEG, 0.05)
        return [synth.spot(t1, 0.0, near(0.3, 0.02), t1, 0.0, near(0.1, 0.02), **warm),
                synth.spot(t2, 0.0, near(0.35, 0.02), t2 - 0.1, 0.0, near(0.2, 0.02), **warm)]
    return [synth.random_spot(rng, log_t) for _ in range(int(rng.integers(1, 3)))]


def _sizes_of_mix(case, k):
    """The k-th member of a served or host batch: the case's sizes are the largest of its mix."""
    div = (1, 2, 4, 8)[k % 4] if case["kind"] == "served" else (1, 2)[k % 2]
    small_e, small_c = max(16, case["energies"] * 3 // 7), max(16, case["channels"] // 5)
    return dict(n_side=max(16, case["n_side"] // div), bins=case["bins"] // (1, 2, 4)[k % 3] or 1,
                energies=case["energies"] if k % 5 < 3 else small_e, channels=case["channels"] if k % 7 < 3 else small_c)


def _params_list(case, seed, ids):
    """The case's parameter sets; `ids(energies, channels)` names its grids and responses."""
    rng = np.random.default_rng([int(seed), 77])
    out = []
    for k in range(case.get("count", 1)):
        s = _sizes_of_mix(case, k) if case["kind"] in ("served", "batch_host") else case
        bb = case.get("atmosphere") == "blackbody"
        g, r = ids(s["energies"], s["channels"])
        log_t, kt = rng.uniform(5.8, 6.6), rng.uniform(0.25, 0.4)
        out.append(synth.params(
            **_star(rng), distance_kpc=0.15, exposure_s=1e6,
            spots=_spots(rng, case["region"], case.get("radius", 0.3), log_t, kt if bb else 0.0),
            atmosphere=_abi.ATM_BLACKBODY if bb else _abi.ATM_NSX, interp=INTERP[case.get("interp", "2l2c_le")],
            beaming=BEAM[case.get("beaming", "iso")], n_side=s["n_side"], n_bins=s["bins"], n_gl=case["nodes"],
            n_fine=3 * s["bins"] if case["nodes"] == 0 else 6 * s["bins"], energy_grid=g, response=r,
            precision=_abi.PREC_FP64 if case.get("precision") == "fp64" else _abi.PREC_FP32,
            fold=FOLD[case.get("fold", "bf16x3")]))
    return out


def _observed(case, seed):
    """Observed counts of a fit: Poisson numbers about a soft pulsed spectrum, none above 0.8 keV."""
    rng = np.random.default_rng([int(seed), 78])
    ch = np.linspace(0.0, 1.0, case["channels"])[:, None]
    ph = np.arange(case["bins"])[None, :] / case["bins"]
    rate = 40.0 * np.exp(-20.0 * ch) * (1.0 + 0.3 * np.cos(2 * np.pi * (ph - 0.2)))
    return rng.poisson(np.where(ch < 0.05, rate, 0.0)).astype(np.float64)


def _fold_flux(case, seed):
    """Spectra to fold, on the device: falling with energy, pulsed, of very different brightness."""
    dev = _dev()
    gen = torch.Generator(device="cpu").manual_seed(int(seed))
    n, b, e = case["count"], case["bins"], case["energies"]
    bright = torch.exp(2.0 * torch.randn(n, 1, 1, generator=gen, dtype=torch.float64))
    slope = 1.0 + 0.5 * torch.rand(n, 1, 1, generator=gen, dtype=torch.float64)
    pulse = 1.0 + 0.5 * torch.rand(n, b, 1, generator=gen, dtype=torch.float64)
    en = torch.from_numpy(_energies(e)).view(1, 1, e)
    alpha = (1e6 / b) * (1.0 + 0.1 * torch.rand(n, generator=gen, dtype=torch.float64))
    flux = (bright * pulse).to(dev) * en.to(dev) * torch.exp(-slope.to(dev) * en.to(dev))
    return flux.contiguous(), alpha.numpy()


# ------------------------------------------------------------------ prepare / run
class _Pool:
    """A batch's device output, handed to torch without a copy; keeps the batch alive with the tensor."""

    def __init__(self, batch, ptr, n):
        self.batch = batch
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": "<f8", "data": (int(ptr), False), "version": 3}


def prepare(case, seed):
    eng = _engine()
    state = dict(case=case, eng=eng)
    if case["kind"] == "fold":
        _, state["rsp"] = _ids(case["energies"], case["channels"])
        state["flux"], state["alpha"] = _fold_flux(case, seed)
        state["counts"] = torch.empty(case["count"], case["channels"], case["bins"], dtype=torch.float64, device="cuda")
        return state
    plist = _params_list(case, seed, _ids)
    state["params"] = plist
    if case["kind"] == "fit":
        state["observed"] = eng.add_observed(plist[0].response, plist[0].n_bins, _observed(case, seed))
    elif case["kind"] == "served":
        state["counts"] = [np.zeros(eng.sizes(p)[1]) for p in plist]
    elif case["kind"] == "batch":
        b = eng.batch(plist)
        state["batch"] = b
        state["flux"] = torch.as_tensor(_Pool(b, b.flux_ptr, b.n_flux), device="cuda")
        state["counts"] = torch.as_tensor(_Pool(b, b.counts_ptr, b.n_counts), device="cuda")
    return state


def _info(info):
    return {k: v for k, v in info.as_dict().items() if k != "status"}


def run(state):
    case, eng = state["case"], state["eng"]
    kind = case["kind"]
    if kind == "profile":
        flux, counts, info = eng.profile(state["params"][0])
        return dict(flux=flux, counts=counts, info=_info(info))
    if kind == "fit":
        fit, info = eng.profile_fit(state["params"][0], state["observed"])
        return dict(fit=fit, info=_info(info))
    if kind == "batch_host":
        flux, counts, infos = eng.profile_batch(state["params"])
        return dict(flux=flux, counts=counts, points=np.array([i.n_points for i in infos]))
    if kind == "served":
        tickets = [eng.submit(p, None, c) for p, c in zip(state["params"], state["counts"])]
        points = []
        for t in tickets:
            points.append(eng.wait(t).n_points)
            eng.release(t)
        return dict(counts=state["counts"], points=np.array(points))
    if kind == "batch":
        state["batch"].launch()
        return dict(flux=state["flux"], counts=state["counts"])
    a = state["alpha"]
    # on the engine's own stream: the flux was made before the call, and nothing else touches the buffers
    _abi.check(_abi.lib().ppm_fold_device(eng.h, state["rsp"], FOLD[case["fold"]], case["count"], case["bins"],
                                          _abi.dptr(a), ctypes.c_void_p(state["flux"].data_ptr()),
                                          ctypes.c_void_p(state["counts"].data_ptr()), None))
    return dict(counts=state["counts"])


# ------------------------------------------------------------------ the work that a pass cannot do without
def _elements(region, radius, n_side):
    """Active surface elements: spot areas over the element area 4 pi / (12 N_side^2)."""
    if region == "point":
        return 1.0
    if region == "cap":
        frac = 0.5 * (1.0 - math.cos(radius))
    elif region == "pair":
        frac = 0.5 * (math.cos(0.1) - math.cos(0.3)) + 0.5 * 0.7 * (1.0 - math.cos(0.35))
    else:
        frac = 0.5 * 0.052 * 0.7 * 1.5  # the prior's mean: radius log-uniform in [0.01, 1], 1.5 spots, 0.7 of a disk
    return max(1.0, 12.0 * n_side * n_side * frac)


def work(case):
    n_tab = 35 * 11 * 166 * 67 * 4.0  # the NSX table in 32 bits
    if case["kind"] == "fold":
        rows = case["count"] * case["bins"]
        return {"bytes": 8.0 * (rows * (case["energies"] + case["channels"]) + case["energies"] * case["channels"]),
                "flops": 2.0 * rows * case["energies"] * case["channels"]}
    nbytes, flops = 0.0, 0.0
    for k in range(case.get("count", 1)):
        s = _sizes_of_mix(case, k) if case["kind"] in ("served", "batch_host") else case
        n_e, n_ch, bins = s["energies"], s["channels"], s["bins"]
        # half of the surface is seen at a time; about 60 operations place a phase point
        points = 0.5 * _elements(case["region"], case.get("radius", 0.3), s["n_side"]) * bins * max(1, case["nodes"])
        if case.get("atmosphere") == "blackbody":
            per_point = 60.0 + 30.0 * n_e
        else:  # a cubic and its sum per energy, 4 mu rows and a cubic per cell of 0.02 dex
            per_point = 60.0 + 8.0 * n_e + 16.0 * (math.log10(E_HI / E_LO) / 0.02 + 4)
        flops += points * per_point + 2.0 * n_ch * n_e * bins
        host = case["kind"] in ("profile", "batch_host")
        out = bins * n_e * (1 if host or case["kind"] == "batch" else 0) + bins * n_ch
        nbytes += 8.0 * (out if case["kind"] != "fit" else 4) + 8.0 * n_e * n_ch * (k == 0)
    if case.get("atmosphere") != "blackbody":
        nbytes += min(n_tab, 16.0 * 166 * 67 * 4 * case.get("count", 1))
    return {"bytes": nbytes, "flops": flops}


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50.0)


# ------------------------------------------------------------------ the same physics in 64 bits
PI = math.pi
C_KM_S = 299792458.0 / 1e3
H_KEV_S, C_CM_S = 4.135668e-18, 299792458.0 * 1e2
IBB = 2.0 / (H_KEV_S ** 3 * C_CM_S ** 2)


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a, dev):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)


def _uniform(x, lo, hi, n):
    """Cell and fraction on a uniform axis, clamped to its ends."""
    t = (x.clamp(lo, hi) - lo) / (hi - lo) * (n - 1)
    i = t.floor().clamp(0, n - 2)
    return i.long(), t - i


def _lagrange(x, nodes):
    """Weights of the cubic through four nodes (last axis) at x."""
    w = []
    for a in range(4):
        v = torch.ones_like(x)
        for b in range(4):
            if a != b:
                v = v * (x - nodes[..., b]) / (nodes[..., a] - nodes[..., b])
        w.append(v)
    return torch.stack(w, -1)


def _bilinear(tab, iu, au, i, a):
    """tab[u][x] at rows iu, au (per ring) and columns i, a (ring x sample)."""
    iu, au = iu[:, None], au[:, None]
    return (1 - au) * ((1 - a) * tab[iu, i] + a * tab[iu, i + 1]) + au * ((1 - a) * tab[iu + 1, i] + a * tab[iu + 1, i + 1])


def _grid(spot, n_side):
    """(cos theta, element solid angle) of the rings with active elements, and ring and azimuth of every element."""
    if spot.kind == _abi.SPOT_POINT:
        return np.array([math.cos(spot.theta1)]), 4 * PI * math.sin(0.5 * spot.angrad1) ** 2, np.zeros(1, int), np.zeros(1)
    n = n_side
    i = np.arange(1, 4 * n)
    ii = np.where(i > 2 * n, 4 * n - i, i)
    z = np.where(ii < n, 1.0 - ii * ii / (3.0 * n * n), 4.0 / 3.0 - 2.0 * ii / (3.0 * n))
    z = np.where(i > 2 * n, -z, z)
    th = np.arccos(z)
    keep = np.abs(th - spot.theta1) <= abs(spot.angrad1) + 2.0 / n  # rings that can touch disk 1
    zs, ring, phis = [], [], []
    for k in np.nonzero(keep)[0]:
        m = int(min(ii[k], n))
        s = 1.0 if ii[k] < n else float((ii[k] - n + 1) % 2)
        phi = PI / (2.0 * m) * (np.arange(1, 4 * m + 1) - s / 2.0)
        c, sn = math.cos(th[k]), math.sin(th[k])
        inside = math.sin(spot.theta1) * sn * np.cos(phi - spot.phi1) + math.cos(spot.theta1) * c > math.cos(spot.angrad1)
        inside &= ~(math.sin(spot.theta2) * sn * np.cos(phi - spot.phi2) + math.cos(spot.theta2) * c > math.cos(spot.angrad2))
        if inside.any():
            ring.append(np.full(int(inside.sum()), len(zs)))
            phis.append(phi[inside])
            zs.append(z[k])
    if not zs:
        return np.zeros(0), PI / (3.0 * n * n), np.zeros(0, int), np.zeros(0)
    return np.array(zs), PI / (3.0 * n * n), np.concatenate(ring), np.concatenate(phis)


def _exact_flux(p, energies):
    """flux[bin][energy] of one parameter set."""
    dev = _dev()
    lens, nsx = _tables()
    if "exact" not in _KEPT:
        _KEPT["exact"] = (_t(lens.ca, dev), _t(lens.lf, dev), _t(lens.cdt, dev),
                          torch.pow(10.0, _t(nsx.log_I, dev)), _t(nsx.mu, dev))
    t_ca, t_lf, t_cdt, t_nsx, t_mu = _KEPT["exact"]
    is_nsx = p.atmosphere == _abi.ATM_NSX
    e = _t(energies, dev)
    out = torch.zeros(p.n_bins, len(energies), dtype=torch.float64, device=dev)
    m, re, nu = p.mass_msun, p.r_eq_km, p.spin_hz
    rs = m * 2.9532501
    x = 0.5 * rs / re
    ob = 2 * PI * nu * math.sqrt(re ** 3 / m) * 2.745011592867327e-6
    o2 = ob * ob * (-0.788 + 1.030 * x)
    logg0 = math.log10(m / (re * re * math.sqrt(1.0 - rs / re))) + math.log10(1.32712440041279419E16)
    d2 = (p.distance_kpc * 3.08567758e+16) ** 2
    co, so = math.cos(p.inclination_rad), math.sin(p.inclination_rad)
    nf = p.n_fine
    k = torch.arange(nf, dtype=torch.float64, device=dev) / nf
    cph, sph = torch.cos(2 * PI * k)[None], torch.sin(2 * PI * k)[None]
    # phase nodes, their bins and weights
    if p.n_gl > 0:
        gx, gw = np.polynomial.legendre.leggauss(p.n_gl)
        lo = np.arange(p.n_bins)[:, None] / p.n_bins
        node = _t((lo + (0.5 + 0.5 * gx[None]) / p.n_bins).ravel(), dev)
        wgt = _t(np.tile(0.5 * gw, p.n_bins), dev)
        nbin = torch.arange(p.n_bins, device=dev).repeat_interleave(p.n_gl)
    else:
        node, wgt = _t(np.arange(p.n_bins) / p.n_bins, dev), torch.ones(p.n_bins, dtype=torch.float64, device=dev)
        nbin = torch.arange(p.n_bins, device=dev)
    for s in range(p.n_spots):
        sp = p.spots[s]
        zs, d_omega, ring, phi = _grid(sp, p.n_side)
        if not len(zs):
            continue
        ct = _t(zs, dev)
        st = torch.sqrt(1 - ct * ct)
        r = re * (1 + o2 * ct * ct)
        u = rs / r
        uu = torch.sqrt(1 - u)
        f = -2 * re * o2 * ct * st / (r * uu)
        ff = torch.sqrt(1 + f * f)
        d_s, cos_tau, sin_tau = r * r * d_omega * ff, 1 / ff, f / ff
        iu, au = _uniform(u, *lens.u[:2], lens.u[2])
        # fine-phase sweep
        col = [v[:, None] for v in (ct, st, r, u, uu, d_s, cos_tau, sin_tau)]
        ct_, st_, r_, u_, uu_, ds_, ctau_, stau_ = col
        cpsi = co * ct_ + so * st_ * cph
        vis = cpsi >= lens.cos_psi[0]
        ic, ac = _uniform(cpsi, *lens.cos_psi[:2], lens.cos_psi[2])
        ca, lf = _bilinear(t_ca, iu, au, ic, ac), _bilinear(t_lf, iu, au, ic, ac)
        sa = torch.sqrt((1 - ca * ca).clamp(min=0))
        saosp = torch.where(cpsi == 1, torch.sqrt(lf), sa / torch.sqrt((1 - cpsi * cpsi).clamp(min=0)))
        csig = ca * ctau_ + saosp * stau_ * (co * st_ - so * ct_ * cph)
        vis &= csig > 0
        beta = 2 * PI * nu * r_ * st_ / uu_ / C_KM_S
        gamma = 1 / torch.sqrt(1 - beta * beta)
        delta = 1 / (gamma * (1 + beta * saosp * so * sph))
        ia, aa = _uniform(ca, *lens.cos_alpha[:2], lens.cos_alpha[2])
        dt1 = _bilinear(t_cdt, iu, au, ia, aa) * r_ / C_KM_S
        dt2 = (re - r_ + rs * torch.log1p((re - r_) / (r_ - rs))) / C_KM_S
        tmp = 2 * sa / torch.sqrt(3 * (1 - u_))
        pp = -tmp * torch.cos((torch.acos((3 * u_ / tmp).clamp(-1, 1)) + 2 * PI) / 3) * r_
        dt2p = (re - pp + rs * torch.log1p((re - pp) / (pp - rs))) / C_KM_S
        dt2 = torch.where(ca >= 0, dt2, 2 * dt2p - dt2)
        csp = csig * delta
        beam = 1.0
        if not is_nsx and p.beaming == _abi.BEAM_SIN2:
            beam = 1 - csp * csp
        elif not is_nsx and p.beaming == _abi.BEAM_COS2:
            beam = csp * csp
        zero = torch.zeros_like(csp)
        fl = torch.where(vis, uu_ * delta ** 3 * csp * lf * (ds_ * gamma) / d2 * beam, zero)
        zz = torch.where(vis, 1 / (delta * uu_), zero)
        ph = torch.where(vis, k[None] + (dt1 + dt2) * nu, zero)
        mu = torch.where(vis, csp, zero)
        # rings whose first or last sample is hidden are skipped; hidden samples are bridged linearly
        live = vis[:, 0] & vis[:, -1]
        idx = torch.arange(nf, device=dev)[None]
        first = torch.where(vis, nf, idx).amin(1)
        last = torch.where(vis, -1, idx).amax(1)
        beg, end = (first - 1).clamp(0, nf - 1)[:, None], (last + 1).clamp(0, nf - 1)[:, None]
        gap = (idx >= first[:, None]) & (idx <= last[:, None])
        frac = (idx - beg).double() / (end - beg).clamp(min=1).double()
        ph = torch.where(gap, ph.gather(1, beg) + (ph.gather(1, end) - ph.gather(1, beg)) * frac, ph)
        zz = torch.where(gap, zz.gather(1, beg) + (zz.gather(1, end) - zz.gather(1, beg)) * frac, zz)
        fl, zz, mu = (torch.cat([v, v[:, :1]], 1) for v in (fl, zz, mu))
        ph = torch.cat([ph, 1 + ph[:, :1]], 1)
        if is_nsx:
            table = _exact_slices(nsx, t_nsx, p.interp, sp.logT, logg0, o2, ob, x, ct, st)
            kt = 10.0 ** sp.logT * 8.617333262E-8
            scale = 10.0 ** (3 * sp.logT) / 6.62607015E-27
        ring_t, phi_t = torch.as_tensor(ring, device=dev), _t(phi, dev)
        keep = live[ring_t]
        ring_t, phi_t = ring_t[keep], phi_t[keep]
        step = max(1, int(6e7 // (len(energies) + 200) // len(node)))
        for j in range(0, len(ring_t), step):
            rg = ring_t[j:j + step].repeat_interleave(len(node))
            q = torch.arange(len(node), device=dev).repeat(len(ring_t[j:j + step]))
            xph = node[q] + phi_t[j:j + step].repeat_interleave(len(node)) / (2 * PI) + 1
            patch = xph - torch.floor(xph)
            patch = torch.where(patch < ph[rg, 0], patch + 1, patch)
            lo_i, hi_i = torch.full_like(rg, -1), torch.full_like(rg, nf + 1)
            for _ in range(nf.bit_length() + 1):  # bisection
                open_ = hi_i - lo_i > 1
                mid = (lo_i + hi_i) >> 1
                right = patch >= ph[rg, mid.clamp(0, nf)]
                lo_i, hi_i = torch.where(open_ & right, mid, lo_i), torch.where(open_ & ~right, mid, hi_i)
            i = lo_i.clamp(0, nf - 1)
            a = (patch - ph[rg, i]) / (ph[rg, i + 1] - ph[rg, i])
            w = (1 - a) * fl[rg, i] + a * fl[rg, i + 1]
            on = w != 0
            rg, q, i, a, w = rg[on], q[on], i[on], a[on], w[on] * wgt[q[on]]
            z = (1 - a) * zz[rg, i] + a * zz[rg, i + 1]
            if is_nsx:
                cs = ((1 - a) * mu[rg, i] + a * mu[rg, i + 1]).clamp(min=float(t_mu[-1]))
                inten = _exact_nsx(nsx, table, rg, p.interp, torch.log10(z / kt)[:, None] + torch.log10(e)[None], cs, t_mu)
                inten = inten * scale
            else:
                ee = z[:, None] * e[None]
                inten = IBB * ee ** 3 / torch.expm1(ee / sp.kT_keV)
            out.index_add_(0, nbin[q], w[:, None] * inten / e[None])
    return out


def _exact_slices(nsx, t_nsx, mode, log_t, logg0, o2, ob, x, ct, st):
    """The NSX table at one temperature and each ring's gravity: [ring][logEkT][mu]."""
    dev = t_nsx.device
    ob2 = ob * ob
    ob4, ob6 = ob2 * ob2, ob2 ** 3
    ce, cp = -0.791 + 0.776 * x, 1.138 - 1.431 * x
    de, fe = -1.315 * x + 2.431 * x * x, -1.172 * x
    dp, fp, d60 = 0.653 * x - 2.864 * x * x, 0.975 * x, 13.47 * x - 27.13 * x * x
    gg = 1 + st * st * (ce * ob2 + de * ob4 + fe * ob6) + ct * ct * (cp * ob2 + dp * ob4 + fp * ob6 - d60 * ob4) \
        + ct.abs() * d60 * ob4
    logg = (torch.log10(gg) + logg0).clamp(*nsx.logg)
    lt = torch.tensor(min(max(log_t, nsx.logT[0]), nsx.logT[1]), dtype=torch.float64, device=dev)
    n_t, n_g = nsx.n[0], nsx.n[1]
    i_t, a_t = _uniform(lt, *nsx.logT, n_t)
    i_g, a_g = _uniform(logg, *nsx.logg, n_g)
    if mode <= 2:
        i_t, i_g = (i_t - 1).clamp(0, n_t - 4), (i_g - 1).clamp(0, n_g - 4)
        off = torch.arange(4, dtype=torch.float64, device=dev)
        w_t = _lagrange(lt, nsx.logT[0] + (nsx.logT[1] - nsx.logT[0]) * (i_t[..., None] + off) / (n_t - 1))
        w_g = _lagrange(logg, nsx.logg[0] + (nsx.logg[1] - nsx.logg[0]) * (i_g[..., None] + off) / (n_g - 1))
    else:
        w_t, w_g = torch.stack([1 - a_t, a_t], -1), torch.stack([1 - a_g, a_g], -1)
    n = w_t.shape[-1]
    at_t = sum(w_t[c] * t_nsx[i_t + c] for c in range(n))
    return sum(w_g[:, c, None, None] * at_t[i_g + c] for c in range(n))


def _exact_nsx(nsx, table, ring, mode, log_ekt, mu, t_mu):
    """Intensity over T^3 of points (ring, mu) at log_ekt[point][energy]."""
    n_e, n_mu = nsx.n[2], nsx.n[3]
    im = (torch.searchsorted(-t_mu, -mu.contiguous(), right=True) - 1).clamp(0, n_mu - 2)
    am = (mu - t_mu[im]) / (t_mu[im + 1] - t_mu[im])
    linear = torch.ones_like(im, dtype=torch.bool) if mode == 4 else \
        (im >= n_mu - 5 if mode in (2, 3) else torch.zeros_like(im, dtype=torch.bool))
    start = torch.where(linear, im.clamp(max=n_mu - 4), (im - 1).clamp(0, n_mu - 4))
    off = torch.arange(4, device=mu.device)
    at = (im - start)[:, None]
    w_lin = torch.where(off == at, (1 - am)[:, None], torch.where(off == at + 1, am[:, None], 0.0))
    w_mu = torch.where(linear[:, None], w_lin, _lagrange(mu, t_mu[start[:, None] + off]))
    rows = sum(w_mu[:, c, None] * table[ring, :, start + c] for c in range(4))  # [point][logEkT]
    lo, hi = nsx.logEkT
    xe = log_ekt.clamp(lo, hi)
    ie, ae = _uniform(xe, lo, hi, n_e)
    if mode == 4:
        return (1 - ae) * rows.gather(1, ie) + ae * rows.gather(1, ie + 1)
    ie = (ie - 1).clamp(0, n_e - 4)
    t = (xe - lo) / (hi - lo) * (n_e - 1) - ie  # cubic through the nodes 0, 1, 2, 3
    val = rows.gather(1, ie) * (-(t - 1) * (t - 2) * (t - 3) / 6)
    val += rows.gather(1, ie + 1) * (t * (t - 2) * (t - 3) / 2)
    val += rows.gather(1, ie + 2) * (-t * (t - 1) * (t - 3) / 2)
    val += rows.gather(1, ie + 3) * (t * (t - 1) * (t - 2) / 6)
    return val.clamp(min=0) if mode == 1 else val


def exact(case, seed):
    if work(case)["flops"] > 4e12:  # beyond about 20 seconds
        return None
    if case["kind"] == "fold":
        flux, alpha = _fold_flux(case, seed)
        rsp = _t(_response(case["energies"], case["channels"]), flux.device)
        return dict(counts=_t(alpha, flux.device)[:, None, None] * torch.matmul(rsp, flux.transpose(1, 2)))
    sizes = {}

    def ids(n_e, n_ch):  # grids and responses by number, without an engine
        sizes.setdefault((n_e, n_ch), len(sizes))
        return sizes[n_e, n_ch], sizes[n_e, n_ch] if n_ch else -1

    plist = _params_list(case, seed, ids)
    by_id = {v: k for k, v in sizes.items()}
    flux, counts = [], []
    for p in plist:
        n_e, n_ch = by_id[p.energy_grid]
        f = _exact_flux(p, _energies(n_e))
        flux.append(f)
        counts.append((p.exposure_s / p.n_bins) * _t(_response(n_e, n_ch), f.device) @ f.T if n_ch else None)
    if case["kind"] == "profile":
        return dict(flux=flux[0], counts=counts[0], info=None)
    if case["kind"] == "fit":
        d, m = _t(_observed(case, seed), counts[0].device), counts[0]
        on = m > 0
        bad = bool(((d != 0) & ~on).any())
        ms = torch.where(on, m, torch.ones_like(m))
        like = torch.where(on, d * torch.log(ms) - m, -m).sum() - torch.lgamma(d + 1).sum()
        return dict(fit=dict(chi2=float((torch.where(on, (d - m) ** 2 / ms, 0.0)).sum() * (1e6 / m.sum())),
                             loglike=-math.inf if bad else float(like), model_total=float(m.sum()), n_zero_model=None),
                    info=None)
    if case["kind"] == "served":
        return dict(counts=counts, points=None)
    if case["kind"] == "batch_host":
        return dict(flux=flux, counts=counts, points=None)
    return dict(flux=torch.cat([f.ravel() for f in flux]), counts=torch.cat([c.ravel() for c in counts]))
