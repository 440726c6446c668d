"""The work a user of this package has it do, as measurable cases.

Every case goes through the package's public entry points (``Context.trace``,
``render``, ``render_batch``, ``adjoint_image``, ``thermal_coefficients`` and
``autograd.IQUVImage``) on seeded synthetic iharm dumps of the sizes that the
tests and the benchmark use.  A program that images a dump keeps one
``Context`` with the dump uploaded and calls it for camera after camera, so
the states of one case share such a session, and what a seed changes is what
changes from call to call: the camera's azimuth, rotation and inclination,
the pixel list, the electron models of a batch, the loss gradient, the fluid
fields of a fit, the plasma parameters of the fits at points.
"""
import math
import os
import tempfile
import weakref

import numpy as np
import torch

import ipole_b200 as ip
from ipole_b200 import autograd, synthdump

# dump name -> (n1, n2, n3, M_unit, R_high).  iharm128 and iharm288 are the
# dumps of the golden images and of the benchmark with their parameters;
# iharm96 has an odd number of azimuthal zones.
DUMPS = {
    "iharm96": (96, 48, 33, 3e27, 20),
    "iharm128": (128, 64, 64, 3e27, 20),
    "iharm288": (288, 128, 128, 7.96e27, 160),
}
BASE = ["--phicam=0", "--MBH=6.5e9", "--dsource=16.8e6", "--fov=160", "--trat_small=1"]

# Costs that the path cannot do without.  A pixel's ray takes about 1300
# steps at the default step size; per step the geodesic executes 1831 FP64
# operations and, at the two thirds of the steps that radiate, the
# coefficients 1535 and the polarized transfer 913 (the unpolarized one a few
# tens).  A refined image traces about a third of its pixels.
STEPS, GEO, COEF, XFER = 1300., 1831., 0.66 * 1535., 0.66 * 913.
REFINED = 0.35


def listed():
    return [
        # a handful of rays: probing pixels of an image, where the latency of
        # the longest ray and the launches are all there is
        {"name": "pixels_16", "kind": "pixels", "dump": "iharm128", "n": 128, "count": 16, "incl": 163, "freq": 230e9},
        # a quick look: an odd-sized adaptively refined thumbnail
        {"name": "refined_33", "kind": "image", "dump": "iharm128", "n": 33, "min": 9, "incl": 60, "freq": 86e9,
         "tier": "fp64", "unpol": False},
        # the ordinary image of the ordinary dump
        {"name": "image_128", "kind": "image", "dump": "iharm128", "n": 128, "min": 0, "incl": 163, "freq": 230e9,
         "tier": "fp64", "unpol": False},
        # a total-intensity image (-unpol), as for light curves
        {"name": "unpol_160", "kind": "image", "dump": "iharm288", "n": 160, "min": 0, "incl": 17, "freq": 230e9,
         "tier": "fp64", "unpol": True},
        # the benchmark's image, FP64 and in the mixed-precision tier
        {"name": "image_400", "kind": "image", "dump": "iharm288", "n": 400, "min": 0, "incl": 163, "freq": 230e9,
         "tier": "fp64", "unpol": False},
        {"name": "mixed_400", "kind": "image", "dump": "iharm288", "n": 400, "min": 0, "incl": 163, "freq": 230e9,
         "tier": "mixed", "unpol": False},
        # a large image refined from a quarter of its resolution
        {"name": "refined_320", "kind": "image", "dump": "iharm288", "n": 320, "min": 80, "incl": 60, "freq": 345e9,
         "tier": "fp64", "unpol": False},
        # electron models of one camera in one call (a parameter sweep)
        {"name": "batch_8x160", "kind": "batch", "dump": "iharm288", "n": 160, "min": 0, "cams": 1, "models": 8,
         "tier": "mixed", "incl": 163},
        # several small refined cameras and models in one call
        {"name": "sweep_3x4x64", "kind": "batch", "dump": "iharm128", "n": 64, "min": 16, "cams": 3, "models": 4,
         "tier": "fp64", "incl": 17},
        # gradients of an image loss with respect to every cell
        {"name": "adjoint_160", "kind": "adjoint", "dump": "iharm288", "n": 160, "incl": 163, "freq": 230e9,
         "ckpt": 16},
        # one step of a fit through torch: forward and backward
        {"name": "fit_40", "kind": "fit", "dump": "iharm128", "n": 40, "incl": 163, "freq": 230e9, "ckpt": 32},
        # the thermal fits alone at given plasma parameters
        {"name": "coefficients_200k", "kind": "coefficients", "count": 200000, "emission": 4, "tier": "fp64"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pixels", "image", "image", "image", "refined", "batch", "adjoint", "fit", "coefficients"])
    dump = rng.choice(["iharm128", "iharm288", "iharm288", "iharm96"])
    incl = rng.choice([17, 60, 120, 163])
    freq = rng.choice([86e9, 230e9, 345e9])
    tier = rng.choice(["fp64", "fp64", "mixed"])
    if kind == "pixels":
        return {"kind": "pixels", "dump": dump, "n": _log(rng, 64, 400), "count": _log(rng, 1, 8000), "incl": incl,
                "freq": freq}
    if kind in ("image", "refined"):
        n = _log(rng, 16, 400)
        unpol = rng.random() < 0.2
        small = max(8, n // 4) if kind == "refined" and n >= 32 else 0
        return {"kind": "image", "dump": dump, "n": n, "min": small, "incl": incl, "freq": freq,
                "tier": "fp64" if unpol else tier, "unpol": unpol}
    if kind == "batch":
        cams, models = rng.randint(1, 3), rng.randint(2, 8)
        n = _log(rng, 24, 240 if cams * models <= 8 else 128)
        return {"kind": "batch", "dump": dump, "n": n, "min": max(8, n // 4) if rng.random() < 0.5 else 0,
                "cams": cams, "models": models, "tier": tier, "incl": incl}
    if kind == "adjoint":
        return {"kind": "adjoint", "dump": dump, "n": _log(rng, 16, 200), "incl": incl, "freq": freq,
                "ckpt": rng.choice([16, 32, 64])}
    if kind == "fit":
        return {"kind": "fit", "dump": rng.choice(["iharm96", "iharm128"]), "n": _log(rng, 16, 80), "incl": incl,
                "freq": freq, "ckpt": 16}
    return {"kind": "coefficients", "count": _log(rng, 100, 1000000), "emission": rng.choice([4, 4, 1]),
            "tier": "fp64"}


# ------------------------------------------------------------------------
# what a program keeps: the loaded dump and a context with it uploaded
# ------------------------------------------------------------------------
_models = {}
_sessions = weakref.WeakValueDictionary()


def _camera_args(case, n, small=0, rot=0., phi=0., incl=None, freq=None):
    a = [*BASE, f"--thetacam={case['incl'] if incl is None else incl}", f"--rotcam={rot}", f"--phicam={phi}",
         f"--freqcgs={case['freq'] if freq is None else freq:.6g}", f"--nx={n}", f"--ny={n}"]
    if small:
        a += [f"--nx_min={small}", f"--ny_min={small}", "--refine_abs=2e-2", "--refine_rel=1e-2"]
    return a


def _model(dump):
    if dump not in _models:
        n1, n2, n3, m_unit, r_high = DUMPS[dump]
        with tempfile.TemporaryDirectory() as td:
            path = os.path.join(td, "dump.ipgc")
            synthdump.write_iharm_dump(path, n1, n2, n3, seed=1)
            p = ip.Params.from_args([f"--dump={path}", *BASE, "--freqcgs=230e9", "--thetacam=163",
                                     f"--M_unit={m_unit:g}", f"--trat_large={r_high}"])
            _models[dump] = ip.Model.load(p)
    return _models[dump]


class _Session:
    """A context with one dump uploaded, in one precision tier."""

    def __init__(self, dump, tier, batch):
        self.ctx = ip.Context(0)
        self.model = _model(dump) if dump else None
        if self.model:
            (self.ctx.upload_batch if batch else self.ctx.upload)(self.model)
        if tier == "mixed":
            self.ctx.set_record_precision(ip.IPG_RECORDS_MIXED)
            self.ctx.set_step_precision(ip.IPG_STEP_FP32)
            self.ctx.set_fit_precision(ip.IPG_FITS_FP32)

    def __del__(self):
        self.ctx.close()


def _session(kind, dump, tier):
    key = (kind, dump, tier)
    s = _sessions.get(key)
    if s is None:
        s = _sessions[key] = _Session(dump, tier, kind == "batch")
    return s


def _points(case, seed):
    """Plasma parameters (nu, ne, Theta_e, B, k-B angle) over the flows' ranges."""
    r = np.random.default_rng(seed)
    n = case["count"]
    return np.stack([10. ** r.uniform(10., 12.5, n), 10. ** r.uniform(2., 7., n), 10. ** r.uniform(-0.5, 2., n),
                     10. ** r.uniform(-1., 2.5, n), np.arccos(r.uniform(-0.999, 0.999, n))], axis=1)


def prepare(case, seed):
    kind = case["kind"]
    r = np.random.default_rng([seed, 7])
    if kind == "coefficients":
        return {"case": case, "session": _session(kind, None, case["tier"]), "points": _points(case, seed)}
    s = _session("batch" if kind == "batch" else kind, case["dump"], case.get("tier", "fp64"))
    model, state = s.model, {"case": case, "session": s}
    n1, n2, n3, m_unit, r_high = DUMPS[case["dump"]]
    rot, phi = r.uniform(-90., 90.), r.uniform(0., 360.)
    incl = case["incl"] + r.uniform(-1., 1.)
    n = case["n"]

    def params(a, mu=m_unit, rh=r_high):
        return ip.Params.from_args([*a, f"--M_unit={mu:.9g}", f"--trat_large={rh:.9g}"])

    if kind == "batch":
        state["params"] = []
        for c in range(case["cams"]):
            inc = (incl + 43. * c) % 180.
            a = _camera_args(case, n, case["min"], rot, phi, inc, (230e9, 86e9, 345e9)[c])
            for k in range(case["models"]):
                state["params"].append(params(a, m_unit * (0.5, 2.)[k % 2] * r.uniform(0.9, 1.1),
                                              (1., 10., 40., 160.)[k // 2] * r.uniform(0.9, 1.1)))
        return state
    p = params(_camera_args(case, n, case.get("min", 0), rot, phi, incl) + (["-unpol"] if case.get("unpol") else []))
    state["params"] = p
    if kind == "pixels":
        at = r.choice(n * n, size=min(case["count"], n * n), replace=False)
        state["ij"] = np.stack([at // n, at % n], axis=1).astype(np.int32)
        state["cam"] = ip.camera_for(p, model.grid)
    elif kind == "adjoint":
        state["dL"] = r.standard_normal((n, n, 4))
    elif kind == "fit":
        fit = autograd.IQUVImage(s.ctx, p, model, case["ckpt"])
        ne, th, b = autograd.derived_fields(fit.prims, m_unit * r.uniform(0.8, 1.2), r_high * r.uniform(0.8, 1.2), 1.)
        state["fit"] = fit
        state["fields"] = [x.cuda() for x in (ne, th, b)]
        state["target"] = torch.from_numpy(r.uniform(0., 1e-3, (n, n, 4))).cuda()
    return state


def _image(img):
    out = {"unpol": img.unpol, "tau": img.tau, "nstep": img.nstep, "oddflag": img.oddflag, "interp": img.interp_flag}
    if img.pol is not None:
        out["pol"] = img.pol
    return out


def run(state):
    case, s = state["case"], state["session"]
    kind = case["kind"]
    if kind == "pixels":
        o = s.ctx.trace(state["cam"], state["ij"])
        return {k: o[k] for k in o.dtype.names}
    if kind == "image":
        return _image(s.ctx.render(state["params"], s.model))
    if kind == "batch":
        imgs = s.ctx.render_batch(state["params"], s.model)
        return {k: np.stack([_image(i)[k] for i in imgs]) for k in ("unpol", "tau", "nstep", "interp", "pol")}
    if kind == "adjoint":
        return s.ctx.adjoint_image(state["params"], s.model, state["dL"], case["ckpt"])
    if kind == "fit":
        f = [x.detach().requires_grad_(True) for x in state["fields"]]
        img = state["fit"](*f)
        ((img - state["target"]) ** 2).sum().backward()
        return {"image": img.detach(), "ne": f[0].grad, "thetae": f[1].grad, "b": f[2].grad}
    return s.ctx.thermal_coefficients(state["points"], case["emission"])


def work(case):
    kind = case["kind"]
    if kind == "coefficients":
        return {"bytes": 17 * 8. * case["count"], "flops": 1200. * case["count"]}
    n1, n2, n3 = DUMPS[case["dump"]][:3]
    cells = float((n1 + 2) * (n2 + 2) * (n3 + 2))
    px = float(case["count"]) if kind == "pixels" else float(case["n"]) ** 2
    # the part of the grid that the rays' gathers can touch
    read = lambda per_cell, rays: per_cell * min(cells, 8. * STEPS * rays)  # noqa: E731
    traced = px * (REFINED if case.get("min") else 1.)
    if kind == "batch":
        k = case["cams"] * case["models"]
        return {"bytes": read(48. + 32. * case["models"], traced * case["cams"]) + 64. * px * k,
                "flops": STEPS * traced * (case["cams"] * GEO + k * (COEF + XFER))}
    flops = STEPS * traced * (GEO + COEF + (0. if case.get("unpol") else XFER))
    if kind in ("adjoint", "fit"):
        # the forward pass, the transfer's and the fits' derivatives (twice
        # their forward cost); the fields in and the gradients out
        passes = 1. if kind == "adjoint" else 2.
        return {"bytes": passes * read(80., px) + 3 * 8. * cells + 96. * px,
                "flops": passes * flops + 2. * STEPS * px * (COEF + XFER)}
    return {"bytes": read(80., traced) + 64. * px, "flops": flops}


# ------------------------------------------------------------------------
# 64-bit values of the fits at points.  The images have none here: a ray is
# a chain of about 1e3-1e4 sequential steps whose finite-difference
# connection (step 1e-7, part of the method) amplifies every rounding, so
# another program's image agrees only to that noise.
# ------------------------------------------------------------------------
EE, CL, ME, HPL = 4.80320680e-10, 2.99792458e10, 9.1093826e-28, 6.6260693e-27


def exact(case, seed):
    if case["kind"] != "coefficients":
        return None
    nu, ne, th, b, ang = _points(case, seed).T
    sth, cth = np.sin(ang), np.cos(ang)
    a = torch.from_numpy(1. / th)
    k0, k1 = (f(a).numpy() for f in (torch.special.modified_bessel_k0, torch.special.modified_bessel_k1))
    k2 = k0 + 2. * th * k1
    x = HPL * nu / (ME * CL * CL * th)
    bnu = (x < 2e-3) * (2 * HPL / CL ** 2 / (x / 24. * (24. + x * (12. + x * (4. + x)))))
    bnu = np.where(x < 2e-3, bnu, 2 * HPL / CL ** 2 / np.expm1(x))
    # Leung, Gammie & Noble 2011: the unpolarized emissivity
    nus = 2. / 9. * EE * b / (2 * np.pi * ME * CL) * th ** 2 * sth
    X = nu / nus
    f = (np.sqrt(X) + 2. ** (11. / 12.) * X ** (1. / 6.)) ** 2
    j = math.sqrt(2.) * np.pi * EE ** 2 * ne * nus / (3. * CL * k2) * f * np.exp(-np.cbrt(X))
    ju = np.where(nu > 1e12 * nus, 0., j) / nu ** 2
    if case["emission"] == 1:
        # Pandya et al. 2016
        nuc = EE * b / (2 * np.pi * ME * CL)
        X = nu / (2. / 9. * nuc * sth * th ** 2)
        pre, t1, ex = ne * EE ** 2 * nuc / CL, math.sqrt(2.) * np.pi / 27. * sth, np.exp(-np.cbrt(X))
        jI = pre * t1 * (np.sqrt(X) + 2. ** (11. / 12.) * X ** (1. / 6.)) ** 2 * ex
        te = th ** (24. / 25.)
        tq = (7. * te + 35.) / (10. * te + 75.)
        jQ = pre * t1 * (np.sqrt(X) + tq * 2. ** (11. / 12.) * X ** (1. / 6.)) ** 2 * ex
        jV = pre * (37. - 87. * np.sin(ang - 28. / 25.)) / (100. * (th + 1.)) * (
            1. + (th ** 0.6 / 25. + 0.7) * X ** (9. / 25.)) ** (5. / 3.) * ex
    else:
        # Dexter 2016
        X = nu / (3. * EE * b * sth / (4. * np.pi * ME * CL) * th ** 2 + 1.)
        c, ex = np.cbrt(X), np.exp(-1.8899 * np.cbrt(X))
        pre = ne * EE ** 2 * nu / (2. * math.sqrt(3.) * CL * th ** 2)
        jI = pre * 2.5651 * (1 + 1.92 / c + 0.9977 / c ** 2) * ex
        jQ = pre * 2.5651 * (1 + 0.93193 / c + 0.499873 / c ** 2) * ex
        jV = 2. * ne * EE ** 2 * nu / (3. * math.sqrt(3.) * CL) * (cth / sth) / th ** 3 * (
            1.81384 / X + 3.42319 / c ** 2 + 0.0292545 / np.sqrt(X) + 2.03773 / c) * ex
    jI, jQ, jV = jI / nu ** 2, jQ / nu ** 2, jV / nu ** 2
    jP = np.hypot(jQ, jV)
    pf = np.where(jI < jP / 0.99, jI / jP * 0.99, 1.)
    jQ, jV = jQ * pf, jV * pf
    # Faraday rotativities: rho_Q of Dexter 2016, rho_V of Shcherbakov 2008
    om0, wp2 = EE * b / (ME * CL), 4. * np.pi * ne * EE ** 2 / ME
    w = 2. * np.pi * nu
    X = th * np.sqrt(math.sqrt(2.) * sth * (1e3 * om0 / w))
    extra = (.011 * np.exp(-X / 47.2) - 2. ** (-1. / 3.) / 3. ** (23. / 6.) * np.pi * 1e4 * (X + 1e-16) ** (-8. / 3.)) * (
        0.5 + 0.5 * np.tanh((np.log(X) - math.log(120.)) / 0.1))
    jf = (2.011 * np.exp(-X ** 1.035 / 4.7) - np.cos(X / 2.) * np.exp(-X ** 1.2 / 2.73) - .011 * np.exp(-X / 47.2)
          + extra)
    rq = w / (2. * CL) * jf * wp2 * om0 ** 2 / w ** 4 * (k1 / k2 + 6. * th) * sth ** 2 * nu
    rv = w / CL * wp2 * om0 / w ** 3 * (k0 / k2 * (1. - 0.11 * np.log(1. + 0.035 * X))) * cth * nu
    z = np.zeros_like(nu)
    return np.stack([ju, ju / bnu, jI, jQ, z, jV, jI / bnu, jQ / bnu, z, jV / bnu, rq, rv], axis=1)
