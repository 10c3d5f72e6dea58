"""Timed workloads of the library: light curves, fits, sampler steps and the
surrogate, called the way a program calls them.

listed() names the workloads, draw() gives one more of the same ranges,
prepare() makes what a program holds before the call, run() makes one call and
work() says what it cannot do without.  exact() computes the same outputs in
plain 64-bit torch and numpy.

Light curves go through host arrays (Model.light_curve, Model.chisq_batch and
chisq_batch_ragged take and return numpy); resident batches keep their data on
the device and take new parameters; the surrogate's calls take device tensors
or host arrays as its own callers hold them.
"""
from __future__ import annotations

import ctypes as C
import importlib
import math

import numpy as np
import torch

lc = importlib.import_module("lcurve-rs_b200")
W = importlib.import_module("lcurve-rs_b200.workloads")
S = importlib.import_module("lcurve-rs_b200.surrogate")

# A posterior of the five fitted parameters (mean, width), as samplers see it.
POST_MEAN = np.array([0.43, 84.0, 0.0157, 28500.0, 4200.0])
POST_SD = np.array([0.065, 1.85, 0.0009, 8000.0, 470.0])


# ---------------------------------------------------------------------------
# the workloads
# ---------------------------------------------------------------------------
def _curve(name, nlat1, nlat2, ntime, ndiv=1, coarse=1, nrad=0, spot=0, extra="none"):
    return dict(name=name, kind="curve", nlat1=nlat1, nlat2=nlat2, ntime=ntime, ndiv=ndiv, coarse=coarse, nrad=nrad,
                spot=spot, extra=extra)


def listed():
    return [
        # the smallest call in use: a model file's default grids (with their
        # coarse copies) at a few dozen times, as when a plot is redrawn
        _curve("curve_tiny", 20, 40, 61, coarse=2),
        # one ordinary light curve: 500 times on the 15,926-element grids
        _curve("curve_small", 50, 100, 500),
        # Doppler beaming of both stars with exposure smearing, odd sizes
        _curve("curve_beamed", 73, 151, 1237, ndiv=3, extra="beam"),
        # a cataclysmic variable: opaque disc with rim, bright spot, irradiation
        _curve("curve_disc", 50, 100, 1000, ndiv=3, nrad=60, spot=100),
        # the large single-model workload at its full size
        _curve("curve_large", 200, 400, 10000, ndiv=5, nrad=200, spot=100),
        # the largest grids (5 million elements) with lensing and star spots,
        # at a tenth of that workload's times
        _curve("curve_lensed", 400, 800, 10000, ndiv=11, nrad=1000, extra="lens"),
        # a fitter's call: 64 parameter sets against one observed light curve
        dict(name="fit_64", kind="fit", nsets=64, nlat1=50, nlat2=100, ntime=500),
        # the headline batch: 1024 uneven models from host arrays
        dict(name="batch_1024", kind="batch", nmodels=1024, nlat1_max=300, nlat2_max=500, ntime_max=5000),
        # one step of the delayed-acceptance sampler: two engine calls for the
        # few walkers that moved (13 of 128 rows)
        dict(name="sampler_13", kind="sampler", rows=13, nphase=256),
        # one step of the plain sampler: two engine calls of 128 rows
        dict(name="sampler_128", kind="sampler", rows=128, nphase=256),
        # one training step of the surrogate network
        dict(name="train_8192", kind="train", batch=8192, width=512, hidden=4, nphase=256),
        # the sampler's screening: two surrogate moves of 128 walkers
        dict(name="screen_128", kind="screen", walkers=128, moves=2, width=512, hidden=4, nphase=256, move="kde"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("curve", "curve", "curve", "fit", "batch", "sampler", "train", "screen"))
    if kind == "curve":
        nlat1 = _log_int(rng, 15, 400)
        case = dict(kind="curve", nlat1=nlat1, nlat2=_log_int(rng, max(20, nlat1), 2 * nlat1 + 20),
                    ntime=_log_int(rng, 30, 10000), ndiv=rng.choice((1, 1, 2, 3, 5, 11)), coarse=rng.choice((1, 1, 2)),
                    nrad=0, spot=0, extra=rng.choice(("none", "none", "beam", "lens")))
        if case["coarse"] == 1 and rng.random() < 0.4:  # a disc's grids come without coarse copies here
            case.update(nrad=_log_int(rng, 20, 400), spot=rng.choice((0, 50, 101)))
        return case
    if kind == "fit":
        nlat1 = _log_int(rng, 20, 100)
        return dict(kind="fit", nsets=_log_int(rng, 1, 200), nlat1=nlat1, nlat2=_log_int(rng, 30, 200),
                    ntime=_log_int(rng, 50, 2000))
    if kind == "batch":
        return dict(kind="batch", nmodels=_log_int(rng, 8, 400), nlat1_max=_log_int(rng, 40, 300),
                    nlat2_max=_log_int(rng, 40, 500), ntime_max=_log_int(rng, 300, 5000))
    if kind == "sampler":
        return dict(kind="sampler", rows=_log_int(rng, 1, 128), nphase=8 * _log_int(rng, 8, 128))
    width, hidden, nphase = 8 * _log_int(rng, 16, 64), rng.randint(2, 4), 8 * _log_int(rng, 8, 64)
    if kind == "train":
        return dict(kind="train", batch=8 * _log_int(rng, 16, 1024), width=width, hidden=hidden, nphase=nphase)
    return dict(kind="screen", walkers=_log_int(rng, 8, 512), moves=rng.randint(1, 4), width=width, hidden=hidden,
                nphase=nphase, move=rng.choice(("kde", "stretch")))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _curve_params(case, seed):
    """The model's parameters as keyword overrides of the base model."""
    rng = np.random.default_rng(seed)
    o = dict(W.SMALL)
    o.update(q=float(rng.uniform(0.1, 0.9)), iangle=float(rng.uniform(77.0, 88.0)), r1=float(rng.uniform(0.008, 0.018)),
             t1=float(rng.uniform(9000.0, 30000.0)), t2=float(rng.uniform(2800.0, 5000.0)))
    n1, n2, k = case["nlat1"], case["nlat2"], case.get("coarse", 1)
    o.update(nlat1f=n1, nlat2f=n2, nlat1c=max(n1 // k, 8), nlat2c=max(n2 // k, 8), phase1=0.0507, phase2=0.4493)
    if case.get("nrad"):
        o.update(add_disc=1, opaque=1, rdisc1=0.02, rdisc2=0.3, texp_disc=-0.75, nrad=case["nrad"], absorb=0.5)
    if case.get("spot"):
        o.update(add_spot=1, temp_spot=12000.0, length_spot=0.05, expon_spot=0.0, epow_spot=2.0, nspot=case["spot"])
    extra = case.get("extra", "none")
    if extra == "beam":
        o.update(beam_factor1=float(rng.uniform(1.0, 2.0)), beam_factor2=float(rng.uniform(1.0, 3.0)),
                 velocity_scale=300.0)
    if extra == "lens":
        o.update(glens1=1, velocity_scale=400.0, tperiod=0.1)
        for s, sign in (("21", 1.0), ("22", -1.0)):
            o[f"stsp{s}_long"] = float(rng.uniform(0.0, 360.0))
            o[f"stsp{s}_lat"] = float(rng.uniform(-90.0, 90.0))
            o[f"stsp{s}_fwhm"] = 10.0
            o[f"stsp{s}_tcen"] = 3500.0 + sign * 500.0
    return o


def _theta(rows, seed):
    rng = np.random.default_rng(seed)
    t = POST_MEAN + POST_SD * rng.standard_normal((rows, 5))
    return np.clip(t, S.PRIOR_LO, S.PRIOR_HI)


def _noise(flux, times, expose, ndiv, seed):
    return W.noisy_data(times, flux, expose, ndiv, seed=seed)


def _fiducial(times, seed, overrides=None):
    """An observed light curve: the fiducial model's fluxes with 1% noise."""
    text = W.model_text(**{**W.SMALL, **(overrides or {})})
    flux = lc.Model(text=text).light_curve(times=times, expose=0.001, ndiv=1).flux
    return _noise(flux, times, 0.001, 1, seed)


def _batch_specs(case, seed):
    """(text, times) of each model: grid sizes and time counts uneven and the
    case's own, physical parameters uniform over the prior box from the seed."""
    size, par, out = np.random.default_rng(case["nmodels"]), np.random.default_rng(seed), []
    for _ in range(case["nmodels"]):
        n1, n2 = (int(size.integers(30, case[k] + 1)) for k in ("nlat1_max", "nlat2_max"))
        theta = dict(zip(S.PARAMS, map(float, par.uniform(S.PRIOR_LO, S.PRIOR_HI))))
        text = W.model_text(**{**W.SMALL, **theta, **dict(nlat1f=n1, nlat1c=n1, nlat2f=n2, nlat2c=n2)})
        out.append((text, np.linspace(-0.2, 0.8, int(size.integers(200, case["ntime_max"] + 1)))))
    return out


def _weights(case, seed):
    """Flat FP32 parameters [W0, b0, W1, b1, ...], He-uniform, small biases."""
    rng = np.random.default_rng(seed)
    sizes = [5] + [case["width"]] * case["hidden"] + [case["nphase"]]
    parts = []
    for i, o in zip(sizes[:-1], sizes[1:]):
        a = math.sqrt(6.0 / i)
        parts += [rng.uniform(-a, a, o * i), rng.uniform(-0.05, 0.05, o)]
    return np.concatenate(parts).astype(np.float32)


def _network(case, seed, max_batch):
    sur = S.Surrogate(n_phase=case["nphase"], width=case["width"], n_hidden=case["hidden"], max_batch=max_batch)
    p = _weights(case, seed)
    lc._capi.check_mlp(sur.L.lcb_mlp_set_params(sur._h, p.ctypes.data_as(C.POINTER(C.c_float)), p.size))
    return sur


def _train_rows(case, seed):
    """Network inputs in [-1, 1] and smooth standardised target curves."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1.0, 1.0, (case["batch"], 5)).astype(np.float32)
    j = np.linspace(0.0, 1.0, case["nphase"], dtype=np.float32)
    basis = np.stack([np.sin(2 * np.pi * (k + 1) * j) for k in range(5)]).astype(np.float32)
    return x, np.ascontiguousarray(x @ basis + 0.1 * x[:, :1] * x[:, 1:2])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "curve":
        model = lc.Model(text=W.model_text(**_curve_params(case, seed)))
        return dict(kind=kind, model=model, times=np.linspace(-0.2, 0.8, case["ntime"]), ndiv=case["ndiv"])
    if kind == "fit":
        times = np.linspace(-0.2, 0.8, case["ntime"])
        grids = dict(nlat1f=case["nlat1"], nlat1c=case["nlat1"], nlat2f=case["nlat2"], nlat2c=case["nlat2"])
        return dict(kind=kind, model=lc.Model(text=W.model_text(**{**W.SMALL, **grids})),
                    data=_fiducial(times, seed, grids), theta=_theta(case["nsets"], seed + 1))
    if kind == "batch":
        specs = _batch_specs(case, seed)
        offs = np.concatenate([[0], np.cumsum([len(t) for _, t in specs])]).astype(np.int64)
        return dict(kind=kind, models=[lc.Model(text=s) for s, _ in specs], offsets=offs,
                    data=_fiducial(np.concatenate([t for _, t in specs]), seed))
    if kind == "sampler":
        setup = S.CurveSetup(n_phase=case["nphase"])
        return dict(kind=kind, engine=S.CurveEngine(setup, _fiducial(setup.times, seed)),
                    halves=(_theta(case["rows"], seed + 1), _theta(case["rows"], seed + 2)))
    if kind == "train":
        sur = _network(case, seed, case["batch"])
        x, y = _train_rows(case, seed + 1)
        return dict(kind=kind, sur=sur, grads=sur._grads_tensor(), x=torch.as_tensor(x).cuda(),
                    y=torch.as_tensor(y).cuda())
    sur = _network(case, seed, 8192)
    sur.sd.fill_(0.1)
    n = case["walkers"]
    rng = np.random.default_rng(seed + 1)
    curve = sur.predict(POST_MEAN[None, :])[0]
    sur.bind_data(_noise(curve, np.linspace(-0.2, 0.8, case["nphase"]), 0.001, 1, seed + 2))
    mcmc = importlib.import_module("lcurve-rs_b200.mcmc")
    walkers, comp = _theta(n, seed + 3), _theta(n, seed + 4)
    ls = -0.5 * sur.chisq(walkers)
    rnd = mcmc.subchain_numbers(rng, case["moves"], n, case["move"])
    return dict(kind=kind, sur=sur, y=walkers, ls=ls, comp=comp, rnd=rnd, move=case["move"])


def run(s):
    kind = s["kind"]
    if kind == "curve":
        r = s["model"].light_curve(times=s["times"], expose=0.001, ndiv=s["ndiv"])
        return dict(flux=r.flux, scalars=np.array([r.wdwarf, r.logg1, r.logg2, r.rv1, r.rv2]))
    if kind == "fit":
        return dict(chisq=s["model"].chisq_batch(s["data"], S.PARAMS, s["theta"], scale=True))
    if kind == "batch":
        chisq, calc, _ = lc.chisq_batch_ragged(s["models"], s["data"], s["offsets"], scale=True, want_calc=True)
        return dict(chisq=chisq, calc=calc)
    if kind == "sampler":
        return dict(chisq=[s["engine"].chisq(t, scale=True) for t in s["halves"]])
    if kind == "train":
        x, y = s["x"], s["y"]
        lc._capi.check_mlp(s["sur"].L.lcb_mlp_train_step(s["sur"]._h, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()),
                                                         x.shape[0], 1e-3, 0.9, 0.999, 1e-8, 0.0))
        with torch.cuda.stream(s["sur"]._stream):  # a copy of its own: the network's buffer goes with the network
            return dict(grads=s["grads"].clone())
    y, ls = s["sur"].subchain(s["y"], s["ls"], s["comp"], s["rnd"], move=s["move"], bandwidth=0.6)
    return dict(y=y, ls=ls)


# ---------------------------------------------------------------------------
# what one pass cannot do without
# ---------------------------------------------------------------------------
def _star_elements(nlat):
    th = (np.arange(nlat) + 0.5) * np.pi / nlat
    return int(np.maximum(16, 2 * nlat * np.sin(th)).astype(np.int64).sum())


def _curve_work(n1, n2, nrad, nspot, nsub, ntime):
    """Flops: 17 per element facing the observer (half of them) and sub-phase;
    and for each element behind the Roche-filling star, two contacts found to
    1e-7 in phase (24 bisection steps of one 22-flop potential each).  Bytes:
    48 of each datum in, 8 out."""
    disc = int(math.pi * nrad * nrad * 1.1) + 20 * nrad if nrad else 0
    elems = n1 + n2 + disc + 2 * nspot
    return dict(flops=8.5 * elems * nsub + 22.0 * 48 * (n1 + disc), bytes=56.0 * ntime)


def work(case):
    kind = case["kind"]
    if kind in ("train", "screen"):
        rows = case["batch"] if kind == "train" else case["walkers"] * case["moves"]
        wts = 5 * case["width"] + case["width"] ** 2 * (case["hidden"] - 1) + case["width"] * case["nphase"]
        if kind == "train":  # forward, input and weight gradients; parameters and both moments in and out
            return dict(flops=6.0 * rows * wts, bytes=rows * 4.0 * (5 + case["nphase"]) + 28.0 * wts)
        return dict(flops=2.0 * rows * wts, bytes=2.0 * wts + 16.0 * case["nphase"] + rows * 8.0 * 13)
    if kind == "sampler":
        one = _curve_work(_star_elements(50), _star_elements(100), 0, 0, case["nphase"], 0)
        n = 2 * case["rows"]
        return dict(flops=n * one["flops"], bytes=n * 48.0)
    if kind == "batch":
        a, b, t = (np.linspace(30, case["nlat1_max"], 9), np.linspace(30, case["nlat2_max"], 9),
                   (200 + case["ntime_max"]) // 2)
        n1 = int(np.mean([_star_elements(int(v)) for v in a]))
        n2 = int(np.mean([_star_elements(int(v)) for v in b]))
        one = _curve_work(n1, n2, 0, 0, t, t)
        return {k: case["nmodels"] * v for k, v in one.items()}
    n1, n2 = _star_elements(case["nlat1"]), _star_elements(case["nlat2"])
    if kind == "fit":
        one = _curve_work(n1, n2, 0, 0, case["ntime"], 0)
        return dict(flops=case["nsets"] * one["flops"], bytes=48.0 * case["ntime"] + 48.0 * case["nsets"])
    return _curve_work(n1, n2, case["nrad"], case["spot"], case["ntime"] * case["ndiv"], case["ntime"])


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------
H, CLIGHT, KB = 6.6262e-34, 2.99792458e8, 1.3806e-23
MOST_EVALS = 1.5e9  # element x sub-phase pairs that plain torch evaluates within seconds


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _planck(wave, temp):
    return 2.0e27 * H * CLIGHT / (torch.exp(1.0e9 * H * CLIGHT / KB / (wave * temp)) - 1.0) / wave ** 3


def _potential(q, secondary, x, y, z):
    """Roche potential of synchronous rotation, in each star's own form."""
    mu = q / (1.0 + q)
    xy = x * x + y * y
    r1, r2 = torch.sqrt(xy + z * z), torch.sqrt(xy + z * z + 1.0 - 2.0 * x)
    own = -(0.5 + 0.5 * xy - x) - (1.0 - mu) * x if secondary else -xy / 2.0 + mu * x
    return -(1.0 - mu) / r1 - mu / r2 + own


def _l1(q):
    mu, lo, hi = q / (1.0 + q), 1e-6, 1.0 - 1e-6
    for _ in range(200):
        x = 0.5 * (lo + hi)
        if (1.0 - mu) / x ** 2 - mu / (1.0 - x) ** 2 - x + mu > 0.0:
            lo = x
        else:
            hi = x
    return 0.5 * (lo + hi)


class _Star:
    """One star's grid in 64 bits: points p, normals d, flux per element.
    Star 1 is a sphere of radius r1, star 2 fills its Roche lobe."""

    def __init__(self, o, star, nlat):
        dev = _dev()
        th = (np.arange(nlat) + 0.5) * np.pi / nlat
        nphi = np.maximum(16, (2.0 * np.pi * np.sin(th) / (np.pi / nlat)).astype(np.int64))
        band = np.repeat(np.arange(nlat), nphi)
        k = np.concatenate([np.arange(n) for n in nphi])
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
        phi = t(2.0 * np.pi * (k + 0.5) / nphi[band])
        ct, st = t(np.cos(th)[band]), t(np.sin(th)[band])
        u = torch.stack([ct, st * torch.cos(phi), st * torch.sin(phi)])
        solid = t((2.0 * np.pi / nphi * np.sin(th) * np.pi / nlat)[band])
        q = o["q"]
        if star == 1:
            rad = torch.full_like(phi, o["r1"])
            self.p, self.d, grav = rad * u, u, torch.ones_like(phi)
        else:
            lobe = 1.0 - _l1(q)
            pot = lambda r: _potential(q, True, 1.0 + r * u[0], r * u[1], r * u[2])  # noqa: E731
            pref = pot(torch.full_like(phi, 1e-3))  # shape only
            l1 = torch.tensor(1.0 - lobe, dtype=torch.float64, device=dev)
            zero = torch.zeros_like(l1)
            pref = _potential(q, True, l1, zero, zero)
            lo, hi = torch.full_like(phi, 0.05 * lobe), torch.full_like(phi, lobe)
            for _ in range(60):
                mid = 0.5 * (lo + hi)
                inside = pot(mid) < pref
                lo, hi = torch.where(inside, mid, lo), torch.where(inside, hi, mid)
            rad = 0.5 * (lo + hi)
            self.p = rad * u
            self.p[0] += 1.0
            g = self._gradient(q, *self.p)
            grav = torch.sqrt((g * g).sum(0))
            self.d = g / grav
            grav = grav / self._back_gravity(q, pref, lobe)
            self.pref, self.lobe = pref, lobe
        area = solid * rad * rad / (u * self.d).sum(0)
        self.flux = area * _planck(550.0, self._temperature(o, star, grav))

    @staticmethod
    def _gradient(q, x, y, z):
        mu = q / (1.0 + q)
        r1, r2 = torch.sqrt(x * x + y * y + z * z), torch.sqrt((x - 1.0) ** 2 + y * y + z * z)
        a, b = (1.0 - mu) / r1 ** 3, mu / r2 ** 3
        return torch.stack([a * x + b * (x - 1.0) - (x - 1.0) + mu - 1.0, a * y + b * y - y, a * z + b * z])

    def _back_gravity(self, q, pref, lobe):
        """|gradient| where the star's surface meets the far side of the axis."""
        dev, lo, hi = pref.device, 0.05 * lobe, lobe
        z = torch.zeros((), dtype=torch.float64, device=dev)
        for _ in range(60):
            mid = 0.5 * (lo + hi)
            if bool(_potential(q, True, z + 1.0 + mid, z, z) < pref):
                lo = mid
            else:
                hi = mid
        g = self._gradient(q, z + 1.0 + 0.5 * (lo + hi), z, z)
        return torch.sqrt((g * g).sum())

    def _temperature(self, o, star, grav):
        t = torch.full_like(grav, o[f"t{star}"])
        if star == 2:
            for s in ("21", "22"):  # Gaussian star spots
                if f"stsp{s}_long" not in o:
                    continue
                lo, la = math.radians(o[f"stsp{s}_long"]), math.radians(o[f"stsp{s}_lat"])
                v = self.p.clone()
                v[0] -= 1.0
                c = (v[0] * math.cos(la) * math.cos(lo) + v[1] * math.cos(la) * math.sin(lo) + v[2] * math.sin(la))
                dist = torch.rad2deg(torch.acos(torch.clamp(c / torch.sqrt((v * v).sum(0)), -1.0, 1.0)))
                sig = o[f"stsp{s}_fwhm"] / 2.3548200450309493
                t = t + (o[f"stsp{s}_tcen"] - t) * torch.exp(-((dist / sig) ** 2) / 2.0)
        base = (t * grav ** o[f"gravity_dark{star}"]) ** 4
        if o["absorb"] == 0.0:
            return base ** 0.25
        v = -self.p.clone()
        v[0] += 1.0 if star == 1 else 0.0
        r = torch.sqrt((v * v).sum(0))
        mu = (self.d * v).sum(0) / r
        rirr = 1.0 - _l1(o["q"]) if star == 1 else o["r1"]
        x0 = torch.clamp(-mu / rirr, -1.0, 1.0)
        part = rirr * (torch.sqrt(1.0 - x0 * x0) * (2.0 + x0 * x0) / 3.0 - x0 * (math.pi / 2 - torch.asin(x0))) / math.pi
        geom = (rirr / r) ** 2 * torch.where(mu >= rirr, mu, torch.where(mu > -rirr, part, torch.zeros_like(mu)))
        return (base + o["absorb"] * o["t2" if star == 1 else "t1"] ** 4 * geom) ** 0.25


def _behind_lobe(q, star2, p, e):
    """Which points p (3 x n) are hidden by the Roche-filling star 2 seen from
    directions e (3 x n): the potential's minimum along the line of sight's
    chord of the lobe's sphere, by sampling and golden-section refinement."""
    d = p.clone()
    d[0] -= 1.0
    b = (e * d).sum(0)
    c = (d * d).sum(0) - star2.lobe ** 2
    disc = b * b - c
    hid = torch.zeros_like(b, dtype=torch.bool)
    idx = torch.nonzero((b < 0.0) & (disc > 0.0)).reshape(-1)
    for part in torch.split(idx, 1 << 20):
        pp, ee = p[:, part], e[:, part]
        far = -b[part] + torch.sqrt(disc[part])
        near = torch.clamp(c[part] / far, min=0.0)
        f = lambda t: _potential(q, True, pp[0] + t * ee[0], pp[1] + t * ee[1], pp[2] + t * ee[2])  # noqa: E731, B023
        best, low = near, f(near)
        for k in range(1, 25):
            t = near + (far - near) * (k / 24)
            v = f(t)
            best, low = torch.where(v < low, t, best), torch.minimum(v, low)
        h = (far - near) / 24
        lo, hi, g = best - h, best + h, (math.sqrt(5.0) - 1.0) / 2.0
        for _ in range(40):
            x1, x2 = hi - g * (hi - lo), lo + g * (hi - lo)
            left = f(x1) < f(x2)
            lo, hi = torch.where(left, lo, x1), torch.where(left, x2, hi)
        hid[part] = torch.minimum(low, f(0.5 * (lo + hi))) < star2.pref
    return hid


def _limb(o, star, mu):
    a = [o.get(f"ldc{star}_{k}", 0.0) for k in (1, 2, 3, 4)]
    m = torch.clamp(mu, 0.0, 1.0)
    x = torch.sqrt(m) if o[f"limb{star}"] == "Claret" else 1.0 - m
    s = x * (a[0] + x * (a[1] + x * (a[2] + x * a[3])))
    return torch.where(mu > 0.0, 1.0 - sum(a) + s if o[f"limb{star}"] == "Claret" else 1.0 - s, torch.zeros_like(mu))


def _star_sum(o, star, grid, star2, phases):
    """The star's summed flux at each phase (no grid interpolation factor)."""
    out = torch.empty_like(phases)
    inc, n = math.radians(o["iangle"]), grid.flux.numel()
    beam, lens = o.get("beam_factor%d" % star, 0.0), star == 2 and o.get("glens1", 0)
    vfac, q = o.get("velocity_scale", 0.0) / (CLIGHT / 1e3), o["q"]
    for at in torch.split(torch.arange(phases.numel(), device=phases.device), max(1, (1 << 23) // n)):
        a = 2.0 * math.pi * phases[at]
        e = torch.stack([math.sin(inc) * torch.cos(a), -math.sin(inc) * torch.sin(a),
                         torch.full_like(a, math.cos(inc))])[:, :, None]
        p, d = grid.p[:, None, :], grid.d[:, None, :]
        mu = (e * d).sum(0)
        see = mu > 0.0
        if star == 2:  # behind the sphere of star 1
            b = (e * p).sum(0)
            see &= ~((b < 0.0) & (b * b - (p * p).sum(0) + o["r1"] ** 2 > 0.0))
        else:
            on = torch.nonzero((see & ((e * p).sum(0) - e[0] < 0.0)).reshape(-1)).reshape(-1)
            hid = _behind_lobe(q, star2, grid.p[:, on % n], e[:, on // n, 0])
            see.reshape(-1)[on[hid]] = False
        c = torch.where(see, mu, torch.zeros_like(mu)) * grid.flux
        if lens:
            gm = (1000.0 * o["velocity_scale"]) ** 3 * o["tperiod"] * 86400.0 / (2.0 * math.pi)
            sep = (gm / (2.0 * math.pi / 86400.0 / o["tperiod"]) ** 2) ** (1.0 / 3.0)
            rl = 4.0 * gm / (1.0 + q) / sep / CLIGHT ** 2
            dist = -(p * e).sum(0)
            w = p + dist * e
            imp = torch.sqrt((w * w).sum(0))
            ph, rd = imp / 2.0, rl * torch.clamp(dist, min=0.0)
            pd = ph + torch.sqrt(ph * ph + rd)
            c = c * torch.where(dist > 0.0, pd * pd / (pd - ph) / ph / 4.0, torch.ones_like(pd))
        if beam:
            vx, vy = -vfac * p[1], vfac * (p[0] - q / (1.0 + q))
            vr = -(e[0] * vx + e[1] * vy)
            c = c * (1.0 - beam * vr) * _limb(o, star, mu - mu * vr - (d[0] * vx + d[1] * vy))
        else:
            c = c * _limb(o, star, mu)
        out[at] = c.sum(1)
    return out


def _exact_curve(o, times, expose, ndiv):
    """Fluxes of a two-star model (no disc) at the times, 64 bits throughout."""
    dev = _dev()
    fine = {1: _Star(o, 1, o["nlat1f"]), 2: _Star(o, 2, o["nlat2f"])}
    coarse = {k: fine[k] if o[f"nlat{k}f"] == o[f"nlat{k}c"] else _Star(o, k, o[f"nlat{k}c"]) for k in (1, 2)}
    k = torch.arange(ndiv, dtype=torch.float64, device=dev)
    t = torch.as_tensor(np.asarray(times), dtype=torch.float64, device=dev)
    step = expose * (k - (ndiv - 1) / 2.0) / max(ndiv - 1, 1) if ndiv > 1 else torch.zeros_like(k)
    ph = (t[:, None] + step[None, :]).reshape(-1)
    pn = ph - torch.floor(ph)
    p1, p2 = o["phase1"], o["phase2"]
    near = (pn <= p1) | (pn >= 1.0 - p1)
    far = ~near & ~(((pn > p1) & (pn < p2)) | ((pn > 1.0 - p2) & (pn < 1.0 - p1)))
    one = lambda s, g, x: float(_star_sum(o, s, g, fine[2], torch.tensor([x], dtype=torch.float64, device=dev))[0])  # noqa: E731, E501
    total = torch.zeros_like(ph)
    for star, use_fine in ((1, near), (2, far)):
        part = torch.empty_like(ph)
        part[use_fine] = _star_sum(o, star, fine[star], fine[2], ph[use_fine])
        rest = ~use_fine
        part[rest] = _star_sum(o, star, coarse[star], fine[2], ph[rest])
        if coarse[star] is not fine[star]:
            lo, hi = 1.0 - 1e-10, 1.0 + 1e-10
            x = pn[rest]
            if star == 1:  # the coarse grid's fluxes meet the fine grid's at phase1
                a, b = (one(1, fine[1], v) / one(1, coarse[1], w)
                        for v, w in ((lo * p1, hi * p1), (1.0 - lo * p1, 1.0 - hi * p1)))
                part[rest] *= (a * (1.0 - p1 - x) + b * (x - p1)) / (1.0 - 2.0 * p1)
            else:          # and star 2's at phase2
                a = one(2, fine[2], 1.0 - hi * p2) / one(2, coarse[2], 1.0 - lo * p2)
                b = one(2, fine[2], hi * p2) / (a * one(2, coarse[2], lo * p2))  # the ratio is taken with a in force
                lower = (b * (p2 - x) + a * (x + p2)) / (2.0 * p2)
                upper = (a * (1.0 + p2 - x) + b * (x - 1.0 + p2)) / (2.0 * p2)
                part[rest] *= torch.where(x < 0.5, lower, upper)
        total += part
    w = torch.ones(ndiv, dtype=torch.float64, device=dev)
    if ndiv > 1:
        w[0] = w[-1] = 0.5
    return ((total.reshape(-1, ndiv) * w).sum(1) / max(1, ndiv - 1)).cpu().numpy()


def _chisq_scaled(calc, data):
    w = data["weight"] / data["ferr"] ** 2
    s = np.sum(w * data["flux"] * calc) / np.sum(w * calc * calc)
    return float(np.sum(w * (data["flux"] - s * calc) ** 2))


def _exact_fit(theta, base, times, data):
    return np.array([_chisq_scaled(_exact_curve({**base, **dict(zip(S.PARAMS, map(float, row)))}, times, 0.001, 1), data)
                     for row in theta])


def _exact_gradients(case, seed):
    """The mean-squared error's gradients, laid out as the network's device buffer
    (the input layer's rows padded with zeros to a multiple of 8)."""
    x, y = (torch.as_tensor(v, dtype=torch.float64, device=_dev()) for v in _train_rows(case, seed + 1))
    flat = torch.as_tensor(_weights(case, seed), dtype=torch.float64, device=_dev())
    sizes, layers, k = [5] + [case["width"]] * case["hidden"] + [case["nphase"]], [], 0
    for i, o in zip(sizes[:-1], sizes[1:]):
        layers.append((flat[k:k + o * i].reshape(o, i).clone().requires_grad_(),
                       flat[k + o * i:k + o * i + o].clone().requires_grad_()))
        k += o * i + o
    a = x
    for n, (w, b) in enumerate(layers):
        a = a @ w.T + b
        if n + 1 < len(layers):
            a = torch.nn.functional.gelu(a)
    ((a - y) ** 2).mean().backward()
    parts = []
    for w, b in layers:
        g = w.grad
        pad = (g.shape[1] + 7) // 8 * 8 - g.shape[1]
        parts += [torch.nn.functional.pad(g, (0, pad)).reshape(-1), b.grad]
    return torch.cat(parts).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "curve":
        n1, n2 = _star_elements(case["nlat1"]), _star_elements(case["nlat2"])
        if case["nrad"] or case["spot"] or (n1 + n2) * case["ntime"] * case["ndiv"] > MOST_EVALS:
            return None  # over 20 s, or a disc whose occultations plain code would have to march rays through
        o = {**dict(nlat1c=case["nlat1"], nlat2c=case["nlat2"]), **_curve_params(case, seed)}
        return dict(flux=_exact_curve(o, np.linspace(-0.2, 0.8, case["ntime"]), 0.001, case["ndiv"]), scalars=None)
    if kind in ("fit", "sampler"):
        rows, nt = (case["nsets"], case["ntime"]) if kind == "fit" else (2 * case["rows"], case["nphase"])
        n1, n2 = case.get("nlat1", 50), case.get("nlat2", 100)
        if rows * nt * (_star_elements(n1) + _star_elements(n2)) > MOST_EVALS:
            return None
        times = np.linspace(-0.2, 0.8, nt)
        grids = dict(nlat1f=n1, nlat1c=n1, nlat2f=n2, nlat2c=n2)
        base = {**W.SMALL, **grids, "phase1": 0.0507, "phase2": 0.4493}
        data = _fiducial(times, seed, grids)  # the observed data are an input
        if kind == "fit":
            return dict(chisq=_exact_fit(_theta(rows, seed + 1), base, times, data))
        return dict(chisq=[_exact_fit(_theta(case["rows"], seed + k), base, times, data) for k in (1, 2)])
    if kind == "train":
        return dict(grads=_exact_gradients(case, seed))
    return None  # a batch of over 20 s; sub-chains whose moves are decisions
