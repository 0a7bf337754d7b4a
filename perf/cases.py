"""The workloads that the performance of this framework is measured on.

Every case is a call that a program makes through the public Python entry points with the
launch configuration the library has by default: propagation of single objects and of whole
populations, with and without the large asteroids; two-body propagation and state-transition
matrices; gradients and sensitivities of an orbit fit; the field checks of a survey; thermal
fluxes; and the joint integration of planets and test particles.  Populations, spans, fields
and geometries have the distributions of the benchmark's configurations.

``listed`` gives the fixed cases, ``draw`` others of the same ranges, ``prepare`` a case's
inputs, ``run`` one pass, ``work`` the bytes and operations a pass cannot do without, and
``exact`` the same outputs from plain 64-bit torch and numpy.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

import kete_b200
from kete_b200 import autodiff, flux, fov, state_transition, synthetic

GM = 0.00029591220828411956
C_INV = 0.005775518331436995  # 1 / c, days per AU
EPOCH = 2460000.5
YEAR = 365.25
OBLIQUITY = 0.40909280422232897
COMET_ROW = (1.0, 0.0, 0.0, 0.0, 0.1112620426, 2.808, 2.15, 5.093, 4.6142, 0.0)
OBSERVER = (0.6, -0.78, 0.0)  # a heliocentric observer for the light delay


def listed():
    return [
        # an ephemeris of one object from host arrays: latency only
        {"name": "nbody_one_1yr", "kind": "nbody", "n": 1, "days": 365.25, "population": "belt",
         "uneven": False, "asteroids": False, "host": True},
        # a catalogue chunk moved to a common epoch
        {"name": "nbody_belt_10k_1yr", "kind": "nbody", "n": 10_000, "days": 365.25,
         "population": "belt", "uneven": False, "asteroids": False, "host": False},
        # the benchmark's default line: a whole population, each object to its own epoch
        {"name": "nbody_mixed_1m_5yr", "kind": "nbody", "n": 1_000_000, "days": 1826.25,
         "population": "mixed", "uneven": True, "asteroids": False, "host": False},
        # the five large asteroids among the perturbers; a ragged count
        {"name": "nbody_asteroids_9973_2yr", "kind": "nbody", "n": 9_973, "days": 730.5,
         "population": "mixed", "uneven": True, "asteroids": True, "host": False},
        # a few objects as an observer sees them (light delay): launch latency
        {"name": "kepler_seen_33", "kind": "kepler", "n": 33, "seen": True},
        # two-body propagation of a population to per-object epochs
        {"name": "kepler_100k", "kind": "kepler", "n": 100_000, "seen": False},
        # covariances of a population through the two-body model
        {"name": "stm_cov_1m", "kind": "stm", "n": 1_000_000},
        # one step of an orbit fit: predicted positions and the gradient of their loss
        {"name": "fit_adjoint_4096", "kind": "fit", "n": 4096, "epochs": 20, "days": 730.5,
         "method": "adjoint"},
        # the sensitivity matrices themselves (differential correction); a ragged count
        {"name": "fit_stm_1021", "kind": "fit", "n": 1021, "epochs": 9, "days": 400.0,
         "method": "stm"},
        # a season of a survey over a population
        {"name": "survey_500k_150_fields", "kind": "survey", "n": 500_000, "fields": 150,
         "days": 45.0},
        # WISE-band fluxes of a catalogue of geometries held on the host
        {"name": "thermal_frm_wise_100k", "kind": "thermal", "n": 100_000, "model": "frm",
         "bands": "wise"},
        # test particles integrated together with the planets
        {"name": "long_2k_10yr", "kind": "long", "n": 2000, "years": 10.0, "batch": 10},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["nbody", "nbody", "nbody", "kepler", "stm", "fit", "survey", "thermal",
                       "long"])
    if kind == "nbody":
        asteroids = rng.random() < 0.25
        n = _log_int(rng, 1, 30_000 if asteroids else 300_000)
        return {"kind": kind, "n": n, "days": round(math.exp(rng.uniform(math.log(20.0),
                                                                         math.log(1826.25))), 3),
                "population": rng.choice(["belt", "mixed"]), "uneven": rng.random() < 0.5,
                "asteroids": asteroids, "host": n < 1000 and rng.random() < 0.5}
    if kind == "kepler":
        return {"kind": kind, "n": _log_int(rng, 1, 1_000_000), "seen": rng.random() < 0.5}
    if kind == "stm":
        return {"kind": kind, "n": _log_int(rng, 1, 1_000_000)}
    if kind == "fit":
        return {"kind": kind, "n": _log_int(rng, 1, 4096), "epochs": rng.randint(2, 20),
                "days": round(rng.uniform(60.0, 730.5), 3), "method": rng.choice(["adjoint", "stm"])}
    if kind == "survey":
        return {"kind": kind, "n": _log_int(rng, 1000, 500_000), "fields": rng.randint(20, 150),
                "days": round(rng.uniform(5.0, 45.0), 3)}
    if kind == "thermal":
        return {"kind": kind, "n": _log_int(rng, 1, 100_000), "model": rng.choice(["neatm", "frm"]),
                "bands": rng.choice(["wise", "neos"])}
    return {"kind": kind, "n": _log_int(rng, 1, 2000), "years": round(rng.uniform(1.0, 10.0), 3),
            "batch": rng.choice([1, 5, 10, 20])}


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
_SPK = []


def _spk_path():
    """The synthetic ephemeris (Sun, planets, Moon, large asteroids), written once."""
    if not _SPK:
        path = os.path.join(tempfile.mkdtemp(prefix="perf_spk_"), "synthetic.bsp")
        synthetic.write_synthetic_spk(path, asteroids=True)
        _SPK.append(path)
    return _SPK[0]


def _load_ephemeris():
    """A program loads its kernels once; ids already loaded are kept."""
    if 10 not in (kete_b200.spice.loaded_ids() if _SPK else ()):
        kete_b200.init()
        kete_b200.spice.kernel_reload([_spk_path()])


def _elements_to_state(a, e, inc, node, argp, mean):
    ecc = torch.where(e < 0.8, mean, torch.full_like(mean, math.pi))
    for _ in range(40):
        ecc = ecc - (ecc - e * torch.sin(ecc) - mean) / (1.0 - e * torch.cos(ecc))
    ce, se = torch.cos(ecc), torch.sin(ecc)
    b = a * torch.sqrt(1.0 - e * e)
    rate = torch.sqrt(GM / a**3) / (1.0 - e * ce)
    x, y, xd, yd = a * (ce - e), b * se, -a * se * rate, b * ce * rate
    cw, sw, co, so = torch.cos(argp), torch.sin(argp), torch.cos(node), torch.sin(node)
    ci, si = torch.cos(inc), torch.sin(inc)
    p = torch.stack([cw * co - sw * so * ci, cw * so + sw * co * ci, sw * si])
    q = torch.stack([-sw * co - cw * so * ci, -sw * so + cw * co * ci, cw * si])
    return (x * p + y * q).contiguous(), (xd * p + yd * q).contiguous()


class _Gen:
    """Seeded draws on the GPU."""

    def __init__(self, seed):
        self.dev = torch.device("cuda", torch.cuda.current_device())
        self.g = torch.Generator(device=self.dev)
        self.g.manual_seed(seed)

    def u(self, n, lo=0.0, hi=1.0):
        return lo + (hi - lo) * torch.rand(n, dtype=torch.float64, device=self.dev, generator=self.g)

    def n(self, *shape):
        return torch.randn(*shape, dtype=torch.float64, device=self.dev, generator=self.g)

    def rayleigh(self, n, sigma):
        return sigma * torch.sqrt(-2.0 * torch.log1p(-self.u(n)))

    def states(self, n, population):
        """Heliocentric ecliptic states: main belt (a U(2.1, 3.3), e Rayleigh 0.1 below 0.4, i
        Rayleigh 10 deg), near-Earth (a U(0.8, 2.5), e U(0.1, 0.7), i Rayleigh 15 deg), or
        nine parts of the one to one of the other."""
        deg, two_pi = math.pi / 180.0, 2.0 * math.pi
        a, e = self.u(n, 2.1, 3.3), torch.clamp(self.rayleigh(n, 0.1), max=0.3999)
        inc = self.rayleigh(n, 10.0 * deg)
        an, en, incn = self.u(n, 0.8, 2.5), self.u(n, 0.1, 0.7), self.rayleigh(n, 15.0 * deg)
        near = self.u(n) < {"belt": -1.0, "neo": 2.0, "mixed": 0.1}[population]
        a, e, inc = torch.where(near, an, a), torch.where(near, en, e), torch.where(near, incn, inc)
        return _elements_to_state(a, e, inc, self.u(n, 0, two_pi), self.u(n, 0, two_pi),
                                  self.u(n, 0, two_pi))

    def comets(self, n, share):
        """Rows of the JPL comet model with A1 ~ N(0, 1e-8), A2 ~ N(0, 1e-9) for a share of
        the objects."""
        has = self.u(n) < share
        row = torch.tensor(COMET_ROW, dtype=torch.float64, device=self.dev)[:, None].repeat(1, n)
        row[1], row[2] = 1e-8 * self.n(n), 1e-9 * self.n(n)
        return torch.where(has, row, torch.zeros_like(row)).contiguous()


def prepare(case, seed):
    _load_ephemeris()
    g, n, kind = _Gen(seed), int(case["n"]), case["kind"]
    s = {"kind": kind, "case": dict(case)}
    if kind == "nbody":
        s["pos"], s["vel"] = g.states(n, case["population"])
        s["ng"] = g.comets(n, 0.05) if case["population"] == "mixed" else None
        s["jd0"] = torch.full((n,), EPOCH, dtype=torch.float64, device=g.dev)
        s["jd1"] = EPOCH + (g.u(n, -case["days"], case["days"]) if case["uneven"]
                            else torch.full_like(s["jd0"], case["days"]))
        if case["host"]:
            for k in ("pos", "vel", "ng", "jd0", "jd1"):
                s[k] = None if s[k] is None else s[k].cpu().numpy()
    elif kind == "kepler":
        s["pos"], s["vel"] = g.states(n, "belt")
        s["jd0"] = torch.full((n,), EPOCH, dtype=torch.float64, device=g.dev)
        s["jd1"] = EPOCH + g.u(n, -1000.0, 1000.0)
        s["obs"] = (torch.tensor(OBSERVER, dtype=torch.float64, device=g.dev) if case["seen"]
                    else None)
    elif kind == "stm":
        s["pos"], s["vel"] = g.states(n, "belt")
        s["jd0"] = torch.full((n,), EPOCH, dtype=torch.float64, device=g.dev)
        s["jd1"] = EPOCH + g.u(n, -1000.0, 1000.0)
        sig = torch.tensor([1e-6] * 3 + [1e-8] * 3, dtype=torch.float64, device=g.dev)
        a = sig[:, None, None] * g.n(6, 6, n)
        s["cov"] = torch.stack([(a[i] * a[:, :]).sum(1) for i in range(6)]).contiguous()
    elif kind == "fit":
        # near-Earth comets and noisy positions of perturbed truth orbits
        s["pos"], s["vel"] = g.states(n, "neo")
        s["a1"], s["a2"] = 1e-8 * g.n(n), 1e-9 * g.n(n)
        s["jd0"] = torch.full((n,), EPOCH, dtype=torch.float64, device=g.dev)
        k = int(case["epochs"])
        s["epochs"] = EPOCH + torch.linspace(case["days"] / k, case["days"], k, dtype=torch.float64,
                                             device=g.dev)
        s["noise"] = 1e-6 * g.n(k, 3, n)
        for name in ("pos", "vel", "a1", "a2"):
            s[name].requires_grad_(True)
    elif kind == "survey":
        s["pos"], s["vel"] = g.states(n, "mixed")
        rng = np.random.default_rng(seed)
        jds = np.sort(EPOCH + rng.uniform(0.0, case["days"], int(case["fields"])))
        lat = np.radians(rng.uniform(-30.0, 30.0, jds.size))
        lon = rng.uniform(0.0, 2.0 * np.pi, jds.size)
        m = 1.7967 + 0.01720209895 * (jds - EPOCH)
        op = np.stack([np.cos(m), np.sin(m), 0.0 * m])
        ov = 0.01720209895 * np.stack([-np.sin(m), np.cos(m), 0.0 * m])
        cols = []
        for i, jd in enumerate(jds):
            pointing = [np.cos(lat[i]) * np.cos(lon[i]), np.cos(lat[i]) * np.sin(lon[i]),
                        np.sin(lat[i])]
            field = fov.RectangleFOV(pointing, 0.0, kete_b200.State("obs", jd, op[:, i], ov[:, i]),
                                     1.8, 1.8)
            cols.append(field.ecliptic_column())
        s["table"] = np.ascontiguousarray(np.stack(cols, axis=1))
    elif kind == "thermal":
        rng = np.random.default_rng(seed)
        r, lon = rng.uniform(1.0, 4.0, n), rng.uniform(0.0, 2.0 * np.pi, n)
        lat = np.clip(rng.normal(0.0, np.radians(15.0), n), -1.4, 1.4)
        s["obj"] = np.ascontiguousarray(np.stack([r * np.cos(lat) * np.cos(lon),
                                                  r * np.cos(lat) * np.sin(lon), r * np.sin(lat)]))
        lo = rng.uniform(0.0, 2.0 * np.pi, n)
        s["obs"] = np.ascontiguousarray(np.stack([np.cos(lo), np.sin(lo), np.zeros(n)]))
        s["pv"] = np.minimum(np.exp(np.log(0.14) + 0.6 * rng.normal(size=n)), 0.9)
        s["h"] = rng.uniform(8.0, 20.0, n)
        s["diam"] = flux.C_V / np.sqrt(s["pv"]) * 10.0 ** (-0.2 * s["h"])
        s["bands"], s["zero"], s["sun"] = _bands(case["bands"])
        s["alb"] = np.ascontiguousarray(np.stack([s["pv"]] * len(s["bands"])))
        s["wise"] = case["bands"] == "wise"
        s["beaming"] = rng.uniform(0.8, 1.4, n)
    else:
        pos, vel = g.states(n, "belt")
        c, sn = math.cos(OBLIQUITY), math.sin(OBLIQUITY)
        rot = torch.tensor([[1, 0, 0], [0, c, -sn], [0, sn, c]], dtype=torch.float64, device=g.dev)
        s["pos"], s["vel"] = (rot @ pos).contiguous(), (rot @ vel).contiguous()
    return s


def _bands(name):
    if name == "wise":
        return (np.array(flux.WISE_BANDS_300K), np.array(flux.WISE_ZERO_MAG_300K),
                np.array(flux.WISE_SUN_CORRECTION))
    return np.array(flux.NEOS_BANDS), np.array(flux.NEOS_ZERO_MAG), np.ones(2)


# ------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    if s["kind"] == "nbody":
        return kete_b200.propagate_n_body_arrays(s["pos"], s["vel"], s["jd0"], s["jd1"],
                                                 include_asteroids=case["asteroids"],
                                                 nongrav=s["ng"])
    if s["kind"] == "kepler":
        return kete_b200.propagate_two_body_arrays(s["pos"], s["vel"], s["jd0"], s["jd1"], s["obs"])
    if s["kind"] == "stm":
        return state_transition.compute_stm_arrays(s["pos"], s["vel"], s["jd0"], s["jd1"],
                                                   covariance=s["cov"])
    if s["kind"] == "fit":
        x = autodiff.nbody_positions(s["pos"], s["vel"], s["a1"], s["a2"], s["jd0"], s["epochs"],
                                     method=case["method"])
        loss = ((x - x.detach() + s["noise"]) ** 2).sum()
        grads = torch.autograd.grad(loss, [s["pos"], s["vel"], s["a1"], s["a2"]])
        return [x.detach(), *grads]
    if s["kind"] == "survey":
        found = fov.fov_state_check_arrays(s["pos"], s["vel"], EPOCH, s["table"])
        return _padded(found, case["n"] * case["fields"] // 1000 + 1024)
    if s["kind"] == "thermal":
        if case["model"] == "neatm":
            return flux.neatm_arrays(s["obj"], s["obs"], s["h"], 0.15, s["diam"], s["pv"],
                                     s["beaming"], 0.9, s["bands"], s["alb"], s["sun"], s["zero"],
                                     s["wise"])
        return flux.frm_arrays(s["obj"], s["obs"], s["h"], 0.15, s["diam"], s["pv"], 0.9, s["bands"],
                               s["alb"], s["sun"], s["zero"], s["wise"])
    return kete_b200.propagate_n_body_long_arrays(s["pos"], s["vel"], EPOCH,
                                                  EPOCH + YEAR * case["years"],
                                                  batch_size=case["batch"])


def _padded(found, room):
    """The detections (field, object, state) in arrays of a length that every seed shares."""
    out_f, out_o = np.full(room, -1, np.int32), np.full(room, -1, np.int32)
    out_s = np.zeros((7, room))
    m = found[0].size
    out_f[:m], out_o[:m], out_s[:, :m] = found
    return out_f, out_o, out_s


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------
# One accepted Radau step: the ephemeris records at its eight times (1,424 operations each with
# ten perturbers), 4.8 corrector iterations of seven force sums (378) and the Radau algebra
# (1,201): 31 thousand operations.  Steps a year: 9 in the belt, 30 near the Earth.
STEP_FLOPS = 8 * 1424 + 4.8 * (7 * 378 + 1201) + 120 + 378
STEPS_YEAR = {"belt": 9.0, "neo": 30.0, "mixed": 11.0}


def work(case):
    n, kind = case["n"], case["kind"]
    if kind == "nbody":
        years = case["days"] / YEAR * (0.5 if case["uneven"] else 1.0)
        steps = n * (4.0 + STEPS_YEAR[case["population"]] * years)
        rows = 80 if case["population"] == "mixed" else 0
        return {"bytes": n * (64 + 52 + rows), "flops": steps * STEP_FLOPS * (1.5 if case["asteroids"]
                                                                             else 1.0)}
    if kind == "kepler":  # four evaluations of the universal Kepler equation and its derivative
        solves = 2 if case["seen"] else 1
        return {"bytes": n * (64 + 60), "flops": n * 600.0 * solves}
    if kind == "stm":  # the solution and six tangents of it, the covariance products
        return {"bytes": n * 8.0 * (8 + 36 + 6 + 72 + 0.5), "flops": n * 2500.0}
    if kind == "fit":
        steps = n * (3.0 * case["epochs"] + STEPS_YEAR["neo"] * case["days"] / YEAR)
        # forward; then the replay with a Jacobian per node and its transposition, or the
        # same Jacobians and eight tangents
        more = 3.0 if case["method"] == "adjoint" else 6.0
        out = n * 8.0 * (3 * case["epochs"] + 8)
        return {"bytes": n * 8.0 * (9 + 3 * case["epochs"]) + out, "flops": steps * STEP_FLOPS * more}
    if kind == "survey":
        chunks = max(1.0, case["days"] / 6.0)
        steps = n * chunks * 5.0
        return {"bytes": n * chunks * 8.0 * 14, "flops": steps * STEP_FLOPS + n * case["fields"] * 60.0}
    if kind == "thermal":  # about 600 facets seen and lit, a black body per band each
        nb = 4 if case["bands"] == "wise" else 2
        return {"bytes": n * 8.0 * (11 + 5 * nb + 2), "flops": n * (2048 * 8.0 + 600 * (30.0 + 35.0 * nb))}
    batches = math.ceil(n / case["batch"])
    bodies = case["batch"] + 9
    steps = batches * (4.0 + 30.0 * case["years"])
    return {"bytes": n * 100.0, "flops": steps * 4.8 * 8 * bodies * 9 * 40.0}


# ------------------------------------------------------------------------------------------
# the same outputs in plain 64-bit arithmetic
# ------------------------------------------------------------------------------------------
def exact(case, seed):
    s = prepare(case, seed)
    if case["kind"] == "nbody":
        return _exact_nbody(case, s)
    if case["kind"] == "kepler":
        p, v = _kepler(s["pos"], s["vel"], s["jd1"] - s["jd0"])
        jd = s["jd1"]
        if s["obs"] is not None:
            dt = -torch.linalg.vector_norm(p - s["obs"][:, None], dim=0) * C_INV
            p, v = _kepler(p, v, dt)
            jd = jd + dt
        return [p, v, jd, None]
    if case["kind"] == "stm":
        dt = s["jd1"] - s["jd0"]
        z = torch.cat([s["pos"], s["vel"]])
        x = _anomaly(s["pos"], s["vel"], dt)
        f = lambda y: torch.cat(_kepler(y[:3], y[3:], dt, x))  # noqa: E731
        cols = [torch.func.jvp(f, (z,), (torch.eye(6, dtype=z.dtype, device=z.device)[i][:, None]
                                         .expand_as(z).contiguous(),))[1] for i in range(6)]
        phi = torch.stack(cols, dim=1)
        tmp = torch.stack([(phi[:, k][:, None] * s["cov"][k][None]) for k in range(6)]).sum(0)
        cov = torch.stack([(tmp[:, k][:, None] * phi[:, k][None]) for k in range(6)]).sum(0)
        y = f(z)
        return [y[:3], y[3:], phi, cov, None]
    if case["kind"] == "thermal":
        return _exact_thermal(case, s)
    return _exact_fit(case, s) if case["kind"] == "fit" else None


def _anomaly(p, v, dt):
    """The change of eccentric anomaly of elliptic two-body motion over dt."""
    r0 = torch.sqrt((p * p).sum(0))
    inv_a = 2.0 / r0 - (v * v).sum(0) / GM
    m = math.sqrt(GM) * inv_a * torch.sqrt(inv_a) * dt
    sig, ec = (p * v).sum(0) / math.sqrt(GM) * torch.sqrt(inv_a), 1.0 - r0 * inv_a
    x = m.clone()
    for _ in range(60):
        f = x + sig * (1.0 - torch.cos(x)) - ec * torch.sin(x) - m
        d = 1.0 + sig * torch.sin(x) - ec * torch.cos(x)
        x = x - torch.clamp(f / d, -1.0, 1.0)
    return x


def _kepler(p, v, dt, x=None):
    """Elliptic two-body motion over dt.  Given the anomaly x, one more Newton step, which
    carries the derivatives with respect to p and v."""
    x = _anomaly(p, v, dt) if x is None else x
    r0 = torch.sqrt((p * p).sum(0))
    inv_a = 2.0 / r0 - (v * v).sum(0) / GM
    a, root_a, root_gm = 1.0 / inv_a, torch.sqrt(1.0 / inv_a), math.sqrt(GM)
    sig, ec = (p * v).sum(0) / root_gm, 1.0 - r0 * inv_a
    m = root_gm * inv_a / root_a * dt
    f = x + (sig / root_a) * (1.0 - torch.cos(x)) - ec * torch.sin(x) - m
    x = x - f / (1.0 + sig / root_a * torch.sin(x) - ec * torch.cos(x))
    c, sn = torch.cos(x), torch.sin(x)
    r = a + (r0 - a) * c + sig * root_a * sn
    half = 2.0 * torch.sin(0.5 * x) ** 2  # 1 - cos
    ff, gd = 1.0 - a / r0 * half, 1.0 - a / r * half
    gg = a * sig / root_gm * half + r0 * root_a / root_gm * sn
    fd = -root_gm * root_a / (r * r0) * sn
    return ff * p + gg * v, fd * p + gd * v


MASSES = {10: 1.0, 5: 0.0009547919099414246, 1: 1.66012082548908e-07, 2: 2.44783828779694e-06,
          399: 3.00348961546514e-06, 301: 3.69430335010988e-08, 4: 3.22715608291416e-07,
          6: 0.00028588567002459455, 7: 4.36624961322212e-05, 8: 5.15138377265457e-05}
ASTEROID_MASSES = {20000001: 4.7191659919436e-10, 20000002: 1.0259143964958e-10,
                   20000004: 1.3026452498655e-10, 20000010: 4.3953391300849e-11,
                   20000704: 1.911e-11}
RADIUS = {10: 0.004654758765894654, 5: 0.00047789450254521576, 399: 4.33036684926559e-05}
J2 = {10: 2.2e-7, 5: 0.014696572, 399: 0.00108262998905}


def _read_spk(path, dev):
    """{body: (centre, start seconds, record length, coefficients (records, 3, k))} of a
    little-endian DAF/SPK with type 2 segments."""
    buf = open(path, "rb").read()
    out, rec = {}, int(np.frombuffer(buf, "<i4", 1, 76)[0])
    while rec:
        off = 1024 * (rec - 1)
        nxt, _, count = np.frombuffer(buf, "<f8", 3, off)
        for k in range(int(count)):
            o = off + 24 + 40 * k
            body, centre, _, _, first, last = np.frombuffer(buf, "<i4", 6, o + 16)
            data = np.frombuffer(buf, "<f8", int(last - first + 1), 8 * (int(first) - 1))
            start, length, size, n_rec = data[-4:]
            coef = data[:-4].reshape(int(n_rec), int(size))[:, 2:].reshape(int(n_rec), 3, -1)
            out[int(body)] = (int(centre), start, length,
                              torch.from_numpy(coef / 149597870.7).to(dev))
        rec = int(nxt)
    return out


def _body(spk, body, t):
    """Barycentric equatorial position and velocity (AU, AU/day) at JD tensor t, last axis 3."""
    centre, start, length, coef = spk[body]
    sec = (t - 2451545.0) * 86400.0 - start
    idx = torch.clamp(torch.floor(sec / length), 0, coef.shape[0] - 1).long()
    x = (2.0 * (sec - idx * length) / length - 1.0)[..., None]
    c = coef[idx]
    t0, t1, u0, u1 = torch.ones_like(x), x, torch.zeros_like(x), torch.ones_like(x)
    p, v = c[..., 0] * t0 + c[..., 1] * t1, c[..., 1] * u1
    for k in range(2, c.shape[-1]):
        t0, t1, u0, u1 = t1, 2 * x * t1 - t0, u1, 2 * t1 + 2 * x * u1 - u0
        p, v = p + c[..., k] * t1, v + c[..., k] * u1
    v = v * (2.0 * 86400.0 / length)
    if centre != 0:
        cp, cv = _body(spk, centre, t)
        p, v = p + cp, v + cv
    return p, v


def _j2_term(rp, r2, radius, j2, gm):
    r = torch.sqrt(r2)
    k = 1.5 * j2 * gm * (radius / r) ** 2 / (r2 * r)
    z2 = 5.0 * (rp[..., 2:3] ** 2) / r2
    return torch.cat([rp[..., :2] * (k * (z2 - 1.0)), rp[..., 2:] * (k * (z2 - 3.0))], dim=-1)


def _force(ids, mass, bp, bv, x, v, ng, rot):
    """spk_accel's model: Newtonian terms, relativistic and J2 terms of Sun and Jupiter, the
    Earth's J2, the JPL comet model.  bp/bv (bodies, nodes, m, 3); x, v (nodes, n, 3)."""
    rp = x[None] - bp
    r2 = (rp * rp).sum(-1, keepdim=True)
    acc = -(rp * (GM * mass[:, None, None, None] / (r2 * torch.sqrt(r2)))).sum(0)
    for k, body in enumerate(ids):
        if body not in J2:
            continue
        gm, rpk, r2k = GM * float(mass[k]), rp[k], r2[k]
        if body == 399:
            acc = acc + _j2_term(rpk, r2k, RADIUS[body], J2[body], gm)
            continue
        rv, r = v - bv[k], torch.sqrt(r2k)
        rel = (4.0 * gm / r - (rv * rv).sum(-1, keepdim=True)) * rpk + \
            4.0 * (rpk * rv).sum(-1, keepdim=True) * rv
        acc = acc + gm * C_INV * C_INV / (r2k * r) * rel
        acc = acc + _j2_term(rpk @ rot, r2k, RADIUS[body], J2[body], gm) @ rot.T
    if ng is not None:
        rs, rv = rp[0], v - bv[0]
        r = torch.sqrt((rs * rs).sum(-1, keepdim=True))
        er = rs / r
        tv = rv - er * (rv * er).sum(-1, keepdim=True)
        et = tv / torch.sqrt((tv * tv).sum(-1, keepdim=True))
        q = r / COMET_ROW[5]
        scale = COMET_ROW[4] * q ** -COMET_ROW[6] * (1.0 + q ** COMET_ROW[7]) ** -COMET_ROW[8]
        acc = acc + scale * (ng[1][:, None] * er + ng[2][:, None] * et)
    return acc


def _exact_nbody(case, s):
    n, days = int(case["n"]), case["days"]
    h_max = 8.0 if case["population"] == "belt" else 1.0
    if days > 800.0 * h_max or n * days / h_max > 8e6:
        return None
    dev = torch.device("cuda", torch.cuda.current_device())
    pos, vel, jd0, jd1, ng = (None if s[k] is None else torch.as_tensor(s[k], device=dev)
                              for k in ("pos", "vel", "jd0", "jd1", "ng"))
    (p, v), = _integrate(pos, vel, jd0, [jd1], h_max, ng, case["asteroids"], not case["uneven"])
    return [p.cpu().numpy(), v.cpu().numpy(), None] if case["host"] else [p, v, None]


def _exact_fit(case, s):
    n = int(case["n"])
    ng = torch.zeros((10, n), dtype=torch.float64, device=s["pos"].device)
    ng[1], ng[2] = s["a1"].detach(), s["a2"].detach()
    ends = [e.expand(n) for e in s["epochs"]]
    got = _integrate(s["pos"].detach(), s["vel"].detach(), s["jd0"], ends, 1.0, ng, False, True)
    return [torch.stack([p for p, _ in got]), None, None, None, None]


def _integrate(pos, vel, jd0, ends, h_max, ng, asteroids, common):
    """Heliocentric ecliptic states at each of the epochs ``ends``: Gauss-Legendre collocation
    (eight nodes, order 16) in equal steps of at most h_max days; ``common``: all objects
    share their epochs."""
    dev = pos.device
    spk = _read_spk(_spk_path(), dev)
    masses = {**MASSES, **(ASTEROID_MASSES if asteroids else {})}
    ids, mass = list(masses), torch.tensor(list(masses.values()), dtype=torch.float64, device=dev)
    c, w = np.polynomial.legendre.leggauss(8)
    c, w = (c + 1.0) / 2.0, w / 2.0
    # integrals of the Lagrange polynomials of the nodes from 0 to each node
    a1 = np.stack([c ** (k + 1) / (k + 1) for k in range(8)], axis=1) @ \
        np.linalg.inv(np.vander(c, increasing=True))
    T = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
    A, AA, B, BB, C = T(a1), T(a1 @ a1), T(w), T(w @ a1), T(c)[:, None]
    co, so = math.cos(OBLIQUITY), math.sin(OBLIQUITY)
    rot = T([[1, 0, 0], [0, co, -so], [0, so, co]])  # ecliptic to equatorial
    sp, sv = _body(spk, 10, jd0)
    x, v = pos.T @ rot.T + sp, vel.T @ rot.T + sv
    out, acc, first = [], None, jd0
    for last in ends:
        steps = int(math.ceil(float((last - first).abs().max()) / h_max)) + 1
        h = (last - first) / steps
        hh = h[:, None]
        acc = None
        for k in range(steps):
            t = first + k * h
            tn = t[None, :1] + C * h[None, :1] if common else t[None] + C * h[None]
            bodies = [_body(spk, b, tn) for b in ids]
            bp, bv = (torch.stack([b[i] for b in bodies]) for i in (0, 1))
            lin = x[None] + C[:, :, None] * (hh * v)[None]
            if acc is None:
                acc = _force(ids, mass, bp, bv, lin, v[None].expand_as(lin), ng, rot)
            for _ in range(12):
                xs = lin + (hh * hh)[None] * torch.einsum("ij,jnc->inc", AA, acc)
                vs = v[None] + hh[None] * torch.einsum("ij,jnc->inc", A, acc)
                acc = _force(ids, mass, bp, bv, xs, vs, ng, rot)
            x = x + hh * v + hh * hh * torch.einsum("j,jnc->nc", BB, acc)
            v = v + hh * torch.einsum("j,jnc->nc", B, acc)
        sp, sv = _body(spk, 10, last)
        out.append((((x - sp) @ rot).T.contiguous(), ((v - sv) @ rot).T.contiguous()))
        first = last
    return out


def _phase_curve(g, phase):
    s, t = np.sin(phase), np.tan(0.5 * phase)
    w = np.exp(-90.56 * t * t)

    def part(a, b, c):
        small = 1.0 - c * s / (0.119 + 1.341 * s - 0.754 * s * s)
        return w * small + (1.0 - w) * np.exp(-a * t ** b)

    return (1.0 - g) * part(3.332, 0.631, 0.986) + g * part(1.862, 1.218, 0.238)


def _exact_thermal(case, s):
    """The facet sum over the 2048-facet lattice, and the reflected light."""
    n, g, emis = int(case["n"]), 0.15, 0.9
    au, pi = 149597870.7, math.pi
    obj, obs, pv, diam = s["obj"], s["obs"], s["pv"], s["diam"]
    r = np.sqrt((obj ** 2).sum(0))
    rel = obj - obs
    d = np.sqrt((rel ** 2).sum(0))
    beam = pi if case["model"] == "frm" else s["beaming"]
    bond = pv * (0.29 + 0.684 * g)
    tss = np.sqrt(np.sqrt((1.0 - bond) * 1360.8 / r ** 2 / (beam * emis * 5.670374419e-8)))
    k = np.arange(2048.0)
    theta, phi = 2.0 * pi * k / 1.618033988749894, np.arccos(1.0 - 2.0 * (k + 0.36) / 2047.72)
    facets = np.stack([np.cos(theta) * np.sin(phi), np.sin(theta) * np.sin(phi), np.cos(phi)])
    dev = torch.device("cuda", torch.cuda.current_device())
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
    F, sun, see, tss_d = T(facets), T(-obj / r), T(rel / d), T(tss)
    lat_f, lat_s = torch.asin(F[2]), torch.asin(sun[2])
    um = [b * 1e-3 for b in s["bands"]]
    thermal = torch.zeros((len(um), n), dtype=torch.float64, device=dev)
    for a in range(0, n, 4096):
        sl = slice(a, a + 4096)
        seen = -(see[:, sl].T @ F)
        lit = (torch.cos(lat_f[None] - lat_s[sl][:, None]) if case["model"] == "frm"
               else sun[:, sl].T @ F)
        lit, seen = torch.clamp(lit, min=0.0), torch.clamp(seen, min=0.0)
        temp = torch.sqrt(torch.sqrt(lit)) * tss_d[sl][:, None]
        on = (temp >= 30.0) & (seen > 0.0)
        temp = torch.where(on, temp, torch.full_like(temp, 100.0))
        for b, wl in enumerate(um):
            ff = 397.289171e17 / wl ** 3 / torch.expm1(1.43877688e4 / (wl * temp))
            if s["wise"]:
                ff = ff * _wise_correction(b, torch.clamp(temp, 100.0, 400.0))
            thermal[b, sl] = torch.where(on, ff * seen, torch.zeros_like(ff)).sum(1)
    thermal = thermal.cpu().numpy() * (emis * pi * (diam / (d * au)) ** 2 / 2048.0)
    phase = np.arccos(np.clip((obj * rel).sum(0) / (r * d), -1.0, 1.0))
    curve = _phase_curve(g, phase)
    dark = phase > 160.0 * pi / 180.0
    hg = np.zeros_like(thermal)
    for b, wl in enumerate(um):
        sunlight = pi * 397.289171e17 / wl ** 3 / np.expm1(1.43877688e4 / (wl * 5778.0)) * \
            (1.3914e6 / au / 2.0 / r) ** 2
        hg[b] = np.where(dark, 0.0, curve * s["alb"][b] * sunlight * (diam / 2.0) ** 2
                         / (d * au) ** 2) * s["sun"][b]
    total = thermal + hg
    vm = np.where(dark, np.nan, s["h"] + 5.0 * np.log10(r * d) - 2.5 * np.log10(curve))
    return {"fluxes": total, "thermal_fluxes": thermal, "hg_fluxes": hg,
            "magnitudes": -2.5 * np.log10(total / s["zero"][:, None]), "v_band_magnitude": vm,
            "v_band_flux": -2.5 * np.log10(vm / 3597.28)}


def _wise_correction(band, t):
    poly = ((-3.78226591e-01, 3.50431748e-03, 1.45866307e-05, -6.67674083e-08, 7.03651986e-11),
            (-8.60229377e-01, 1.54988562e-02, -5.10705456e-05, 7.68314436e-08, -4.32238900e-11),
            (-1.29814355e+00, 2.43268763e-02, -9.05178737e-05, 1.50095351e-07, -9.35433316e-11),
            (2.17247804e+01, -1.46084733e+01, 3.85364000e+00, -4.51512551e-01, 1.98397252e-02))
    x = t if band < 3 else torch.log(t)
    v = sum(c * x ** k for k, c in enumerate(poly[band]))
    return 1.0 / v if band < 3 else v
