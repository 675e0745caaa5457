"""Performance cases of the photon trace, its batched and differentiable
forms and the event-coordinate pass, through the package's public calls.

The sizes run from an interactive call (a thousand photons) to the full
workloads of ``marx_gb300.workloads`` (1e7 to 2e7 photons), the 256-source
batch, the 4e6-ray gradient step and 1e7 events.  Inputs are made on the GPU
from a seed, with the workloads' own distributions.

``exact`` restates in 64-bit torch, from the calibration data alone, what
has a closed form: the aspect dither, the mirror with blur, scattering and
struts and the ACIS-I chips of the grating-less workloads, the weighted-ray
image and its gradient (by automatic differentiation), and the focal-plane
and sky coordinates of events (in the well-conditioned form of the sky
angles).  The gratings, the HRC and the pulse-height response have no such
restatement here: their outputs are held against an earlier build's.
"""
import math
import os
import struct
import tempfile

import numpy as np
import torch

from marx_gb300 import batched as B
from marx_gb300 import diff as D
from marx_gb300 import events as E
from marx_gb300 import workloads as W
from marx_gb300._native import DevicePhotons, Engine
from marx_gb300.caldb.pack import DEFAULT_PACK, pack_with_fef
from marx_gb300.photons import PhotonList

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FEF_FILE = os.path.join(ROOT, "tests", "golden", "acis_fef_synthetic.fits")
ARCSEC = math.pi / 648000.0
DEV = "cuda"

# Floating-point operations per photon (ray) of the path, counted over
# samples of each workload with a counting arithmetic on the host
# restatement (LETG and HRC by comparison with the HETG and ACIS ones).
FLOPS = {"plain_onaxis": 333, "plain_scatter": 558, "plain_hetg": 620, "plain_letg": 640, "plain_hrci": 560,
         "letg_hrcs": 660, "batch": 380, "ray": 327, "event": 150}
# Columns of a photon in and out: energy, p, time, flags, tag; x, p, flags,
# shell, order, chip, pixels, dither state.
PHOTON_BYTES = 48 + 75
EXTRA_BYTES = {"plain_letg": 4, "plain_hrci": 2, "letg_hrcs": 15}
BASE = ("x", "p", "flags", "mirror_shell", "order", "ccd_num", "y_pixel", "z_pixel", "dither_state")
EXTRA = {"plain_letg": ("support_orders",), "plain_hrci": ("pulse_height",),
         "letg_hrcs": ("support_orders", "pulse_height", "u_pixel", "v_pixel", "detector_region")}


def listed():
    return [
        # an interactive call or one small source: launches and latency count
        {"name": "scatter_1k", "kind": "trace", "workload": "plain_scatter", "n": 1000},
        # a short grating exposure, ragged, below the size that takes the wavefront kernels
        {"name": "hetg_48k", "kind": "trace", "workload": "plain_hetg", "n": 48611},
        # the on-axis configuration at its own size
        {"name": "onaxis_1m", "kind": "trace", "workload": "plain_onaxis", "n": 1_000_000},
        # the scattered, dithered ACIS-I field: the headline configuration
        {"name": "scatter_10m", "kind": "trace", "workload": "plain_scatter", "n": 10_000_000},
        # the HETG spectrum on ACIS-S: the largest plain configuration
        {"name": "hetg_20m", "kind": "trace", "workload": "plain_hetg", "n": 20_000_000},
        # LETG with its supports, Drake flat and HRC-S, ragged
        {"name": "letg_hrcs_4m", "kind": "trace", "workload": "letg_hrcs", "n": 3_999_971},
        # ACIS with its pulse-height response in the tables, as an observer runs it
        {"name": "scatter_fef_2m", "kind": "fef", "workload": "plain_scatter", "n": 2_000_000},
        # the C host path: page-locked host columns in and out
        {"name": "host_1m", "kind": "host", "workload": "plain_scatter", "n": 1_000_003},
        # 256 uneven sources in one launch
        {"name": "batch_256", "kind": "batch", "sources": 256, "nmax": 1_000_000},
        # one optimisation step of the mirror geometry: image, loss, gradient
        {"name": "gradient_4m", "kind": "gradient", "n": 4_000_000},
        # marx2fits' event columns of a long ACIS-I observation
        {"name": "events_10m", "kind": "events", "n": 10_000_000, "pixadj": "EDSER"},
        # a whole observation: source photons, trace, pruning, event columns
        {"name": "observe_1m", "kind": "observe", "workload": "plain_hetg", "n": 1_000_003},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | rng.randint(0, 1)

    kind = rng.choice(["trace", "trace", "trace", "trace", "fef", "host", "batch", "gradient", "events", "observe"])
    if kind == "trace":
        name = rng.choice(["plain_onaxis", "plain_scatter", "plain_hetg", "plain_letg", "plain_hrci", "letg_hrcs"])
        return {"kind": kind, "workload": name, "n": size(700, 12_000_000 if name in W.PLAIN else 4_000_000)}
    if kind == "fef":
        return {"kind": kind, "workload": rng.choice(["plain_scatter", "plain_hetg"]), "n": size(20_000, 4_000_000)}
    if kind == "host":
        return {"kind": kind, "workload": rng.choice(["plain_scatter", "plain_hetg"]), "n": size(5000, 2_000_000)}
    if kind == "batch":
        return {"kind": kind, "sources": rng.randint(8, 256), "nmax": size(10_000, 1_000_000)}
    if kind == "gradient":
        return {"kind": kind, "n": size(50_000, 4_000_000)}
    if kind == "events":
        return {"kind": kind, "n": size(2000, 10_000_000), "pixadj": rng.choice(["EDSER", "RANDOMIZE", "NONE", "EXACT"])}
    return {"kind": kind, "workload": rng.choice(["plain_hetg", "plain_scatter"]), "n": size(20_000, 4_000_000)}


# ------------------------------------------------------------------ inputs --
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _inputs(name, n, seed):
    """energy (n), p (3, n) and arrival times of a workload's photons."""
    g = _gen(seed)
    rand = lambda m=n: torch.rand(m, generator=g, device=DEV, dtype=torch.float64)  # noqa: E731
    p = torch.zeros(3, n, device=DEV, dtype=torch.float64)
    if name == "plain_onaxis":
        p[0] = -1.0
        return torch.full((n,), 1.49, device=DEV, dtype=torch.float64), p, torch.zeros(n, device=DEV, dtype=torch.float64)
    if name in ("plain_scatter", "plain_hrci"):
        energy = torch.exp(math.log(0.3) + rand() * math.log(8.0 / 0.3))
        theta, phi = rand() * (600.0 * ARCSEC), rand() * (2 * math.pi)
        st = torch.sin(theta)
        p[0], p[1], p[2] = -torch.cos(theta), st * torch.cos(phi), st * torch.sin(phi)
        return energy, p, rand() * 1e4
    # absorbed power law on 0.4-8 keV, photon index 1.7, NH = 1e21 / cm^2
    p[0] = -1.0
    a, kept, have = -0.7, [], 0
    while have < n:
        m = int((n - have) * 1.6) + 1024
        e = (0.4 ** a + rand(m) * (8.0 ** a - 0.4 ** a)) ** (1.0 / a)
        e = e[rand(m) < torch.exp(-1e21 * W.SIGMA_1KEV * e ** (-8.0 / 3.0))]
        kept.append(e)
        have += e.numel()
    return torch.cat(kept)[:n].contiguous(), p, rand() * 1e4


_fef = []   # the table pack with the pulse-height response, written once


def _fef_pack():
    if not _fef:
        _fef.append(tempfile.TemporaryDirectory())
        pack_with_fef(DEFAULT_PACK, FEF_FILE, os.path.join(_fef[0].name, "fef.mxpack"))
    return os.path.join(_fef[0].name, "fef.mxpack")


def _photons(name, n, seed):
    d = DevicePhotons(n)
    d.energy, d.p, d.arrival_time = _inputs(name, n, seed)
    d.tag = torch.arange(n, device=DEV, dtype=torch.int32)
    return d


def _pinned(name, n, seed):
    """A host photon list in page-locked memory, and its torch columns."""
    d = _photons(name, n, seed)
    host, cols = PhotonList.__new__(PhotonList), {}
    host.n = n
    for k in ("energy", "p", "arrival_time", "flags", "tag", *BASE):
        if k not in cols:
            cols[k] = getattr(d, k).cpu().pin_memory()
            a = cols[k].numpy()
            setattr(host, k, a.view(np.uint32) if k in ("flags", "tag") else a)
    return host, cols


def _sources(case, seed):
    """Point sources with the case's photon counts, gratings and detectors
    in directions and energy bands of the seed's."""
    src = B.batched_sources(nsrc=case["sources"], nmax=case["nmax"])
    r = np.random.default_rng(seed)
    for s in src:
        th, phi = r.uniform(0.0, 600.0 * ARCSEC), r.uniform(0.0, 2 * math.pi)
        s.p[:] = [-math.cos(th), math.sin(th) * math.cos(phi), math.sin(th) * math.sin(phi)]
        s.energy_min, s.energy_max = r.uniform(0.3, 1.0), r.uniform(5.0, 10.0)
    return src


def _theta(seed):
    return np.random.default_rng(seed + 17).normal(0.0, 0.3, D.NPARAM)


def _event_columns(n, seed):
    g = _gen(seed)
    rand = lambda: torch.rand(n, generator=g, device=DEV)  # noqa: E731
    t = torch.sort(torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * (n / 30 * E.ACIS_FRAME_TIME)).values.float()
    return {"ccd": torch.randint(0, 4, (n,), generator=g, device=DEV, dtype=torch.int8), "xpixel": rand() * 1024,
            "ypixel": rand() * 1024, "time": t, "sky_ra": (8 * ARCSEC * torch.sin(t / 159.0)).float(),
            "sky_dec": (8 * ARCSEC * torch.sin(t / 112.5)).float(), "sky_roll": torch.full((n,), 4.137, device=DEV),
            "b_energy": 0.3 + 9.7 * rand()}


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "seed": seed}
    if kind in ("trace", "fef", "host"):
        w = W.ALL[case["workload"]]()
        s["engine"] = Engine(w.cfg, pack=_fef_pack() if kind == "fef" else None)
        s["columns"] = BASE + (("pulse_height", "pi") if kind == "fef" else EXTRA.get(case["workload"], ()))
        if kind == "host":
            s["photons"], s["cols"] = _pinned(case["workload"], case["n"], seed)
            s["p0"] = s["cols"]["p"].clone()
        else:
            s["photons"] = _photons(case["workload"], case["n"], seed)
            s["p0"] = s["photons"].p.clone()
    elif kind == "batch":
        s["engine"] = Engine(B.batched_config())
        s["sources"] = _sources(case, seed)
        s["batch"] = B.Batch(s["engine"], s["sources"])
    elif kind == "gradient":
        s["engine"] = Engine(D.diff_mirror_config())
        w = D.diff_workload(n_rays=case["n"], seed=seed & 0xFFFF)
        s["diff"] = D.DiffImage.centred(s["engine"], w.cfg)
        c = s["diff"].cfg.copy()
        c.seed = w.target_seed
        other = D.DiffImage(s["engine"], c)
        s["target"] = other.forward(w.theta_true, D.FRESH).clone()
        torch.cuda.synchronize()
        other.close()
        s["theta"] = _theta(seed)
    elif kind == "events":
        s["engine"] = Engine(W.plain_scatter().cfg)
        s["events"], s["n"] = _event_columns(case["n"], seed), case["n"]
        s["params"] = E.params(roll_nom=237.36968458476, pixel_adjust=case["pixadj"])
    else:
        w = W.ALL[case["workload"]]()
        s["engine"], n = Engine(w.cfg), case["n"]
        th = 40.0 * ARCSEC
        s["source"] = B.make_source((-math.cos(th), math.sin(th), 0.0), "GAUSS", (2.0,), energy=(0.5, 7.0), num_photons=n)
        s["photons"] = DevicePhotons(n)
        s["times"] = torch.sort(torch.rand(n, generator=_gen(seed), device=DEV, dtype=torch.float64) * 1e4).values
        s["params"] = E.params(roll_nom=w.cfg.roll_nom)
        # the observation's event list: columns with room for every photon
        s["list"] = {k: torch.zeros(n, device=DEV, dtype=getattr(torch, np.dtype(t).name)) for k, t in E.OUTPUTS.items()}
        s["list"]["index"] = torch.zeros(n, device=DEV, dtype=torch.int32)
    return s


# ------------------------------------------------------------------- passes --
def run(s):
    kind, eng = s["kind"], s["engine"]
    if kind in ("trace", "fef"):
        d = s["photons"]
        d.p.copy_(s["p0"])       # the trace replaces directions and flags in place
        d.flags.zero_()
        eng.trace(d, seed=s["seed"])
        return {k: getattr(d, k) for k in s["columns"]}
    if kind == "host":
        s["cols"]["p"].copy_(s["p0"])
        s["cols"]["flags"].zero_()
        eng.trace_host(s["photons"], seed=s["seed"])
        return {k: s["cols"][k] for k in s["columns"]}
    if kind == "batch":
        s["batch"].run(s["seed"])
        out = s["batch"].photons()
        for t in out.values():
            t.owner = s["batch"]     # the columns are views of the batch's memory
        return out
    if kind == "gradient":
        d = s["diff"]
        image = d.forward(s["theta"], D.RECORD)
        loss, dl = d.mse(image, s["target"])
        return {"image": image, "loss": loss, "dl": dl, "gradient": d.adjoint(s["theta"], dl)}
    if kind == "events":
        return E.event_coords(eng, s["params"], s["events"], s["n"], seed=s["seed"])
    d = s["photons"]
    B.generate_source(eng, s["source"], 0, s["seed"], d)
    d.arrival_time.copy_(s["times"])
    eng.trace(d, seed=s["seed"])
    index = eng.compact(d.flags)
    ev = dict(E.photon_events(d, index), b_energy=d.energy.float())
    out = dict(E.event_coords(eng, s["params"], ev, index.numel(), seed=s["seed"]), index=index)
    for k, v in out.items():
        s["list"][k][:index.numel()] = v
    return s["list"]


def work(case):
    kind = case["kind"]
    if kind in ("trace", "fef", "host", "observe"):
        name, n = case["workload"], case["n"]
        more = EXTRA_BYTES.get(name, 0) + (6 if kind == "fef" else 0)
        return {"bytes": n * (PHOTON_BYTES + more), "flops": n * FLOPS[name]}
    if kind == "batch":
        mean = (case["nmax"] - 1e3) / math.log(case["nmax"] / 1e3)   # of a log-uniform count
        return {"bytes": case["sources"] * mean * (PHOTON_BYTES - 20), "flops": case["sources"] * mean * FLOPS["batch"]}
    if kind == "gradient":
        return {"bytes": 2 * case["n"] + 4 * 256 * 256 * 8, "flops": 2 * case["n"] * FLOPS["ray"]}
    return {"bytes": case["n"] * 85, "flops": case["n"] * FLOPS["event"]}


# ------------------------------------------- the path in 64-bit arithmetic --
def _tables():
    """The calibration pack's sections, read as plain data."""
    b = open(DEFAULT_PACK, "rb").read()
    out = {}
    for i in range(struct.unpack_from("<I", b, 8)[0]):
        name, dt, nd, *rest = struct.unpack_from("<48sII4QQQ", b, 16 + 104 * i)
        kind = ("<f4", "<f8", "<i4")[dt]
        a = np.frombuffer(b, kind, rest[5] // int(kind[2]), rest[4]).reshape(rest[:nd])
        out[name.rstrip(b"\0").decode()] = torch.from_numpy(a.copy()).to(DEV)
    return out


def _philox(seed, tag, slot, domain):
    m32 = 0xFFFFFFFF
    c = [tag.to(torch.int64), torch.full_like(tag, slot, dtype=torch.int64), torch.full_like(tag, domain, dtype=torch.int64),
         torch.zeros_like(tag, dtype=torch.int64)]
    k0, k1 = seed & m32, (seed >> 32) & m32
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
        a, b = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57     # modulo 2^64
        c = [((b >> 32) & m32) ^ c[1] ^ k0, b & m32, ((a >> 32) & m32) ^ c[3] ^ k1, a & m32]
    return c


def _uniform(seed, tag, slot, domain=0x5A5A0001):
    c = _philox(seed, tag, slot, domain)
    return ((c[0] << 21) | (c[1] >> 11)).double() * 2.0 ** -53


def _normal(seed, tag, slot):
    """The single-precision Box-Muller normal, operation by operation."""
    c = _philox(seed, tag, slot, 0x5A5A0002)
    f = np.float32
    u1, u2 = ((c[0] >> 8) + 1).float() * 2.0 ** -24, (c[1] >> 8).float() * 2.0 ** -24
    m, e = torch.frexp(u1)
    m, e = m * 2, (e - 1).float()
    big = m > float(f(1.41421356))
    m, e = torch.where(big, m * 0.5, m), e + big.float()
    s = (m - 1) / (m + 1)
    s2 = s * s
    poly = torch.full_like(s, float(f(0.0909090909)))
    for k in (0.111111111, 0.142857143, 0.2, 0.333333333):
        poly = float(f(k)) + s2 * poly
    log = e * float(f(0.693145752)) + (e * float(f(1.42860677e-06)) + (2 * s) * (1 + s2 * poly))
    x4 = u2 * 4
    q = x4.floor()
    t = (x4 - q) * float(f(1.57079632679))
    t2 = t * t
    cs, sn = torch.full_like(t, float(f(2.08767570e-09))), torch.full_like(t, float(f(1.60590438e-10)))
    for k in (-2.75573192e-07, 2.48015873e-05, -1.38888889e-03, 4.16666667e-02, -0.5, 1.0):
        cs = float(f(k)) + t2 * cs
    for k in (-2.50521084e-08, 2.75573192e-06, -1.98412698e-04, 8.33333333e-03, -1.66666667e-01, 1.0):
        sn = float(f(k)) + t2 * sn
    sn = t * sn
    return (torch.sqrt(-2 * log) * torch.where(q == 0, cs, torch.where(q == 1, -sn, torch.where(q == 2, -cs, sn)))).double()


def _interp(x, xp, yp):
    """Linear interpolation of a float table, rounded to float."""
    k = torch.searchsorted(xp, x).clamp(max=xp.numel() - 1)
    j = (k - 1).clamp(min=0)
    k = j + 1
    x0 = xp[j].double()
    slope = (yp[k] - yp[j]).double() / (xp[k].double() - x0)
    return torch.where(x == xp[k], yp[k], (yp[j].double() + slope * (x.double() - x0)).float())


def _shells(cfg, T, theta):
    """The four shells' conics, frames, apertures: theta moves them."""
    rdb, out, total = T["hrma/rdb"].cpu().numpy().reshape(2, 4, 9), [], 0.0
    one, zero = torch.ones((), device=DEV, dtype=torch.float64), torch.zeros((), device=DEV, dtype=torch.float64)

    def about_z(a):
        c, s = torch.cos(a), torch.sin(a)
        return torch.stack([torch.stack([c, -s, zero]), torch.stack([s, c, zero]), torch.stack([zero, zero, one])])

    def about(n, a):
        c, s = torch.cos(a), torch.sin(a)
        x = torch.stack([torch.stack([zero, -n[2], n[1]]), torch.stack([n[2], zero, -n[0]]), torch.stack([-n[1], n[0], zero])])
        return c * torch.eye(3, device=DEV, dtype=torch.float64) + (1 - c) * torch.outer(n, n) + s * x

    for i in range(4):
        sh = {"cap": cfg.hrma_cap_x + cfg.shell_xoffset[i], "optic": []}
        for o in range(2):
            x0, y0, z0, p, k, rho, az, el, length = (float(v) for v in rdb[o, i])
            to = torch.stack([one * (z0 - sh["cap"]), -(x0 + theta[4 * i + 2] * 1e-3), y0 + theta[4 * i + 3] * 1e-3])
            az, el = -(az + theta[4 * i] / 3600) * (math.pi / 180), -(el + theta[4 * i + 1] / 3600) * (math.pi / 180)
            rz = about_z(-az)
            fwd, bwd = about(rz[:, 1], -el) @ rz, about_z(az) @ about(rz[:, 1], el)
            sh["optic"].append({"a": 1.0 - p, "b": -2.0 * k, "c": rho * rho, "half": 0.5 * length, "to": to, "fwd": fwd, "bwd": bwd})
        q, half = sh["optic"][0], sh["optic"][0]["half"]
        sh["front"] = sh["cap"] - float(rdb[0, i, 2]) + half
        r = [math.sqrt(q["c"] + x * (q["b"] + x * (q["a"] - 1))) for x in (-half, half)]
        sh["rmin"], sh["rmax"] = r[0] - 2 * half * math.tan(0.67 * math.pi / 180), r[1]
        total += (sh["rmax"] - sh["rmin"]) * (sh["rmax"] + sh["rmin"])
        sh["fraction"] = total
        out.append(sh)
    for sh in out:
        sh["fraction"] /= total
    return out


def _dot(a, b):
    return (a * b).sum(0)


def _unit(a):
    return a / torch.sqrt(_dot(a, a))


def _conic(q, x, p):
    """Hit mask, position and unit normal of rays on a conic."""
    x = x + (-x[0] / p[0]) * p
    alpha, beta = q["a"] * p[0] * p[0] - 1, q["b"] * p[0] - 2 * (p[1] * x[1] + p[2] * x[2])
    gamma = q["c"] - x[1] * x[1] - x[2] * x[2]
    disc = beta * beta - 4 * alpha * gamma
    real = disc.detach() > 0
    root = beta + torch.where(beta < 0, -1.0, 1.0) * torch.sqrt(torch.where(real, disc, 1.0))
    tp, tm = -2 * gamma / root, -0.5 * root / alpha
    inside = lambda t: real & (p[0] * t >= -q["half"]) & (p[0] * t < q["half"])  # noqa: E731
    okp, okm = inside(tp), inside(tm)
    t = torch.where(okp & ~(okm & (p[0] * tm > p[0] * tp)), tp, tm)
    x = torch.stack([p[0] * t, x[1] + p[1] * t, x[2] + p[2] * t])
    return okp | okm, x, _unit(torch.stack([(q["a"] - 1) * x[0] + 0.5 * q["b"], -x[1], -x[2]]))


def _reflectivity(cos, beta, delta):
    """Fresnel reflectivity, mean of both polarisations, index 1 - delta + i beta."""
    sr, si = (1 - delta) ** 2 - beta ** 2, 2 * (1 - delta) * beta
    wr, wi = cos * cos - (delta * (2 - delta) + beta * beta), si     # n^2 - sin^2
    r = torch.sqrt(wr * wr + wi * wi)
    big = torch.sqrt(0.5 * (r + wr.abs()))
    rr, ri = torch.where(wr >= 0, big, 0.5 * wi / big), torch.where(wr >= 0, 0.5 * wi / big, big)
    perp = ((cos - rr) ** 2 + ri ** 2) / ((cos + rr) ** 2 + ri ** 2)
    par = ((cos * sr - rr) ** 2 + (cos * si - ri) ** 2) / ((cos * sr + rr) ** 2 + (cos * si + ri) ** 2)
    return 0.5 * (perp + par)


STRUT_X = ((1492.060, 942.266), (0.5 * 1.965 * 25.4, -0.5 * 1.965 * 25.4), (-1050.353, -1271.333))
STRUT_W = (0.25 * 25.4, 0.375 * 25.4, 0.25 * 25.4)


def _struts(cfg, k, x, p):
    hit = torch.zeros(x.shape[1], device=DEV, dtype=torch.bool)
    for plane in STRUT_X[k]:
        t = (plane + cfg.hrma_cap_x - x[0]) / p[0]
        y, z = x[1] + t * p[1], x[2] + t * p[2]
        for i in range(3):
            if i:
                y, z = math.cos(math.pi / 6) * y - math.sin(math.pi / 6) * z, math.sin(math.pi / 6) * y + math.cos(math.pi / 6) * z
            hit |= (y.abs() < STRUT_W[k]) | (z.abs() < STRUT_W[k])
    return hit


def _scatter(T, table, energy, sin_alpha, r):
    """The scattering angle of a WFold table at (energy sin alpha, r)."""
    hdr, theta = T[table + "/hdr"].double().reshape(-1, 7), T[table + "/theta"].double()
    theta = theta.reshape(hdr.shape[0], -1)
    ea, num = hdr[:, 0].contiguous(), hdr.shape[0]
    i = torch.searchsorted(ea, energy * sin_alpha).clamp(1, num - 1)

    def at(a):
        h = hdr[a]
        d = (r - h[:, 1]) / h[:, 2]
        k = d.clamp(min=0).floor().clamp(max=theta.shape[1] - 2).long()
        k = torch.minimum(k, h[:, 6].long() - 1)
        nxt = torch.minimum(k + 1, h[:, 6].long() - 1)
        v = torch.where(k + 1 >= h[:, 6].long(), theta[a, k], (1 - (d - k)) * theta[a, k] + (d - k) * theta[a, nxt])
        v = torch.where(r > h[:, 3], (h[:, 4] * (1 - r)).clamp(min=1e-300) ** h[:, 5], v)
        return torch.where(r < h[:, 1], 0.0, v)

    t0, t1 = at(i - 1), at(i)
    return t0 + (t1 - t0) * (energy * sin_alpha - ea[i - 1]) / (ea[i] - ea[i - 1])


def _aperture(shells, seed, tag):
    pick, r = _uniform(seed, tag, 1), _uniform(seed, tag, 2)
    shell = (pick[None] >= torch.tensor([s["fraction"] for s in shells], device=DEV, dtype=torch.float64)[:, None]).sum(0)
    return shell, r, 2 * math.pi * (_uniform(seed, tag, 3) - 0.125)


def _trace_plain(cfg, energy, p, time, seed):
    """x, p, pixels and dither state of photons with no grating on ACIS-I."""
    T, n = _tables(), energy.numel()
    tag = torch.arange(n, device=DEV)
    out = {"x": torch.zeros(3, n, device=DEV, dtype=torch.float64), "p": p.clone()}
    for k in ("y_pixel", "z_pixel"):
        out[k] = torch.zeros(n, device=DEV, dtype=torch.float64)
    out["dither_state"] = dith = torch.zeros(3, n, device=DEV, dtype=torch.float64)
    if cfg.dither:
        blur = cfg.aspect_blur * ARCSEC
        for k in range(2):
            dith[k] = (cfg.dither_amp[k] * ARCSEC * torch.sin(2 * math.pi * time / cfg.dither_period[k] + cfg.dither_phase[k])).float()
        roll = math.fmod(math.radians(cfg.roll_nom), 2 * math.pi)
        dith[2] = float(np.float32(roll - 2 * math.pi if roll >= math.pi else roll))
        c, s = torch.cos(dith[2]), torch.sin(-dith[2])
        p = torch.stack([p[0], c * p[1] - s * p[2], c * p[2] + s * p[1]])
        ra, dec = dith[0] + blur * _normal(seed, tag, 0), dith[1] + blur * _normal(seed, tag, 1)
        ny, nz = torch.sin(dec), -torch.cos(dec) * torch.sin(ra)
        d = 2 * torch.sin(0.5 * dec) ** 2 + torch.cos(dec) * 2 * torch.sin(0.5 * ra) ** 2      # 1 - cos dec cos ra
        k = (p[1] * ny + p[2] * nz) / (2 - d)
        p = torch.stack([p[0] + (ny * p[2] - nz * p[1] - d * p[0]), p[1] + (k * ny + nz * p[0] - d * p[1]),
                         p[2] + (k * nz - ny * p[0] - d * p[2])])
    shells = _shells(cfg, T, torch.zeros(18, device=DEV, dtype=torch.float64))
    shell, ur, angle = _aperture(shells, seed, tag)
    optc = T["hrma/optconst"].reshape(3, -1)
    fe = energy.float()
    beta, delta = _interp(fe, optc[0], optc[1]).double(), _interp(fe, optc[0], optc[2]).double()
    for i, sh in enumerate(shells):
        k = (shell == i).nonzero().squeeze(1)
        sid, slot, blocked = (1, 3, 4, 6)[i], 4, None
        e, q = energy[k], p[:, k]
        corr = T["hrma/corr%d" % sid].reshape(2, -1)
        scale = torch.sqrt(_interp(fe[k], corr[0], corr[1]).double())
        r0, r1 = sh["rmin"], sh["rmax"]
        rad = torch.sqrt(r0 * r0 + (r1 * r1 - r0 * r0) * ur[k]) if cfg.aperture_area_uniform else r0 + (r1 - r0) * ur[k]
        to = sh["optic"][0]["to"]
        x = torch.stack([torch.full_like(rad, sh["front"]), rad * torch.sin(angle[k]) - to[1], rad * torch.cos(angle[k]) - to[2]])
        bad = _struts(cfg, 0, x, q) if cfg.use_struts else torch.zeros_like(rad, dtype=torch.bool)

        def keep(mask, *v):
            """Photons outside mask end here, with x and q as they are."""
            out["x"][:, k[~mask]], out["p"][:, k[~mask]] = x[:, ~mask], q[:, ~mask]
            return [a[..., mask] for a in v]

        for o, opt in enumerate(sh["optic"]):
            x, q = opt["fwd"] @ (x + opt["to"][:, None]), opt["fwd"] @ q
            hit, at, nrm = _conic(opt, x, q)
            e, scale, bad, at, nrm, x, q, k = keep(hit, e, scale, bad, at, nrm, x, q, k)
            x = at
            if cfg.use_blur:
                length = torch.sqrt(nrm[1] ** 2 + nrm[2] ** 2)
                phi = 2 * math.pi * _uniform(seed, k, slot)
                ang = (cfg.blur_p[i], cfg.blur_h[i])[o] * ARCSEC * _normal(seed, k, 2 + o)
                slot += 1
                w = torch.stack([torch.cos(phi) * length, (torch.sin(phi) * nrm[2] - torch.cos(phi) * nrm[0] * nrm[1]) / length,
                                 (-torch.sin(phi) * nrm[1] - torch.cos(phi) * nrm[0] * nrm[2]) / length])
                nrm = torch.cos(ang) * nrm + torch.sin(ang) * w
            pn = _dot(q, nrm)
            ok = _uniform(seed, k, slot) < _reflectivity(pn.abs(), beta[k], delta[k]) * scale
            slot += 1
            e, scale, bad, nrm, pn, x, q, k = keep(ok, e, scale, bad, nrm, pn, x, q, k)
            q = q - 2 * pn * nrm
            if cfg.use_wfold:
                dg = _scatter(T, "wfold/%s%d" % ("ph"[o], sid), e, -pn, _uniform(seed, k, slot)) * (cfg.scat_p[i], cfg.scat_h[i])[o]
                ok = dg <= math.pi / 4
                e, scale, bad, nrm, dg, x, q, k = keep(ok, e, scale, bad, nrm, dg, x, q, k)
                dg = torch.where(_uniform(seed, k, slot + 1) < 0.5, -dg, dg)
                slot += 2
                q = _unit(torch.cos(dg) * q + torch.sin(dg) * (nrm - _dot(q, nrm) * q))
            x, q = opt["bwd"] @ x - opt["to"][:, None], opt["bwd"] @ q
            if cfg.use_struts:
                ok = _struts(cfg, 1 + o, x, q)
                if o == 0:
                    e, scale, bad, x, q, k = keep(~ok, e, scale, bad, x, q, k)
                else:
                    bad = bad | ok
        (k, x, q), _ = keep(~bad, k, x, q), None
        _acis_i(cfg, T, seed, k, x, q, time[k], out)
    return out


def _chips(T):
    geom, ofs = T["acis/geom"].reshape(-1, 13), T["acis/aimpt_i"].reshape(-1)[:3] + T["acis/origin"].reshape(-1)[:3]
    for c in range(4):
        row = geom[(geom[:, 0] == c).nonzero().max()]
        ll, xh, yh = row[1:4] + ofs, row[4:7] - row[1:4], row[7:10] - row[1:4]
        xl, yl = torch.linalg.vector_norm(xh), torch.linalg.vector_norm(yh)
        yield c, ll, xh / xl, yh / yl, xl, yl


def _acis_i(cfg, T, seed, k, x, p, time, out):
    free = torch.ones_like(k, dtype=torch.bool)
    out["x"][:, k], out["p"][:, k] = x, p
    for _, ll, xh, yh, xl, yl in _chips(T):
        nrm = torch.linalg.cross(xh, yh)
        r = x - ll[:, None]
        r = r - ((nrm @ r) / (nrm @ p)) * p
        dx, dy = xh @ r, yh @ r
        on = free & (dx >= 0) & (dx < xl) & (dy >= 0) & (dy < yl)
        free &= ~on
        xpix, ypix = (dx / (xl / 1024)).float().double(), (dy / (yl / 1024)).float().double()
        frame = cfg.acis_exposure_time + cfg.acis_frame_transfer_time
        late = on & (torch.fmod(time, frame) > cfg.acis_exposure_time)
        at = r + ll[:, None]
        ypix = torch.where(late, (1 + 1022 * _uniform(seed, k, 14)).float().double(), ypix)
        row = ll[:, None] + xh[:, None] * (xpix * (xl / 1024)) + yh[:, None] * (ypix * (yl / 1024))
        at = torch.where(late, row, at)
        aim = torch.tensor([cfg.focal_length, 0.0, 0.0], device=DEV, dtype=torch.float64)[:, None]
        q = torch.where(late, _unit(at - aim), p)
        i = k[on]
        out["x"][:, i], out["p"][:, i] = at[:, on], q[:, on]
        out["y_pixel"][i], out["z_pixel"][i] = xpix[on], ypix[on]


class _Rays:
    """The weighted rays of one seed and their focal-plane image."""

    def __init__(self, cfg, n, seed, energy, src):
        self.cfg, self.n, self.seed, self.src, self.T = cfg, n, seed, src, _tables()
        fe = torch.tensor([energy], device=DEV, dtype=torch.float64).float()
        o = self.T["hrma/optconst"].reshape(3, -1)
        self.beta, self.delta = _interp(fe, o[0], o[1]).double(), _interp(fe, o[0], o[2]).double()
        self.corr = []
        for sid in (1, 3, 4, 6):
            c = self.T["hrma/corr%d" % sid].reshape(2, -1)
            self.corr.append(torch.sqrt(_interp(fe, c[0], c[1]).double()))

    def trace(self, theta, lo, hi):
        """Focal-plane y, z and weight of the rays lo..hi that reach it."""
        shells, tag = _shells(self.cfg, self.T, theta), torch.arange(lo, hi, device=DEV)
        shell, ur, angle = _aperture(shells, self.seed, tag)
        angles = (self.src + theta[16:18]) * ARCSEC
        p0 = _unit(torch.cat([-torch.ones(1, device=DEV, dtype=torch.float64), -torch.tan(angles)])[:, None])
        got = []
        for i, sh in enumerate(shells):
            k = (shell == i).nonzero().squeeze(1)
            rad = sh["rmin"] + (sh["rmax"] - sh["rmin"]) * ur[k]
            to, p, w = sh["optic"][0]["to"], p0.expand(3, k.numel()), torch.ones_like(rad)
            x = torch.stack([torch.full_like(rad, sh["front"]), rad * torch.sin(angle[k]) - to[1], rad * torch.cos(angle[k]) - to[2]])
            ok = ~_struts(self.cfg, 0, x.detach(), p.detach())
            x, p, w = x[:, ok], p[:, ok], w[ok]
            for o, opt in enumerate(sh["optic"]):
                x, p = opt["fwd"] @ (x + opt["to"][:, None]), opt["fwd"] @ p
                hit, x, nrm = _conic(opt, x, p)
                x, p, nrm, w = x[:, hit], p[:, hit], nrm[:, hit], w[hit]
                pn = _dot(p, nrm)
                w = w * _reflectivity(pn.abs(), self.beta, self.delta) * self.corr[i]
                p = p - 2 * pn * nrm
                x, p = opt["bwd"] @ x - opt["to"][:, None], opt["bwd"] @ p
                ok = ~_struts(self.cfg, 1 + o, x.detach(), p.detach())
                x, p, w = x[:, ok], p[:, ok], w[ok]
            got.append(torch.stack([x[1] - x[0] / p[0] * p[1], x[2] - x[0] / p[0] * p[2], w]))
        return torch.cat(got, 1)

    def image(self, theta, centre, lo, hi, pitch=0.024, sigma=1.0, side=256):
        y, z, w = self.trace(theta, lo, hi)
        u, v = (y - centre[0]) / pitch + 0.5 * side - 0.5, (z - centre[1]) / pitch + 0.5 * side - 0.5
        uc, vc = (u.detach() + 0.5).floor(), (v.detach() + 0.5).floor()
        norm = 1 / (math.sqrt(2 * math.pi) * sigma)
        taps = torch.arange(-5, 6, device=DEV, dtype=torch.float64)
        ku = norm * torch.exp(-0.5 * ((taps[:, None] - (u - uc)) / sigma) ** 2)
        kv = norm * torch.exp(-0.5 * ((taps[:, None] - (v - vc)) / sigma) ** 2)
        flat = torch.zeros(side * side, device=DEV, dtype=torch.float64)
        for a in range(11):
            row = vc.long() + a - 5
            col = uc.long()[None] + torch.arange(-5, 6, device=DEV)[:, None]
            ok = (row >= 0) & (row < side) & (col >= 0) & (col < side)
            flat = flat.index_add(0, (row * side + col)[ok], (w * kv[a] * ku)[ok])
        return flat.reshape(side, side) / self.n

    def chunks(self):
        return [(lo, min(self.n, lo + (1 << 19))) for lo in range(0, self.n, 1 << 19)]


def _exact_gradient(case, seed):
    w, cfg = D.diff_workload(n_rays=case["n"], seed=seed & 0xFFFF), D.diff_mirror_config()
    src = torch.tensor([w.cfg.src_y, w.cfg.src_z], device=DEV, dtype=torch.float64)
    vec = lambda t: torch.tensor(np.asarray(t), device=DEV, dtype=torch.float64)  # noqa: E731
    rays = _Rays(cfg, case["n"], w.cfg.seed, w.cfg.energy, src)
    with torch.no_grad():
        m = [rays.trace(vec(np.zeros(18)), lo, hi) for lo, hi in rays.chunks()]
        total = sum(float(a[2].sum()) for a in m)
        centre = [sum(float((a[2] * a[k]).sum()) for a in m) / total for k in range(2)]
        del m
        other = _Rays(cfg, case["n"], w.target_seed, w.cfg.energy, src)
        target = sum(other.image(vec(w.theta_true), centre, lo, hi) for lo, hi in other.chunks())
        theta = vec(_theta(seed))
        image = sum(rays.image(theta, centre, lo, hi) for lo, hi in rays.chunks())
    dl = 2 * (image - target) / image.numel()
    grad = torch.zeros_like(theta)
    for lo, hi in rays.chunks():
        t = theta.clone().requires_grad_(True)
        grad += torch.autograd.grad(rays.image(t, centre, lo, hi), t, dl)[0]
    return {"image": image, "loss": ((image - target) ** 2).mean(), "dl": dl, "gradient": grad.cpu().numpy()}


FLIGHT_GRADES = ((10, 11, 138, 139), (2, 34, 130, 162), (18, 22, 50, 54), (8, 12, 136, 140), (0, 0, 0, 0),
                 (16, 17, 48, 49), (72, 76, 104, 108), (64, 65, 68, 69), (80, 81, 208, 209))


def _exact_events(case, seed):
    T, n, ev = _tables(), case["n"], _event_columns(case["n"], seed)
    k = torch.arange(n, device=DEV)
    u = [_uniform(seed, k, j, 0x5A5A0004) for j in range(3)]
    chip = [ev["xpixel"] + 1.0, ev["ypixel"] + 1.0]
    frame = (ev["time"].double() / E.ACIS_FRAME_TIME).long()
    start = torch.cat([torch.ones(1, device=DEV, dtype=torch.bool), frame[1:] != frame[:-1]])
    first = torch.cummax(torch.where(start, k, 0), 0).values if case["pixadj"] != "EXACT" else k
    ra, dec, roll = (ev[c].double()[first] for c in ("sky_ra", "sky_dec", "sky_roll"))
    sub = [(3 * (c.double() - c.double().floor())).long() for c in chip]
    grade = torch.tensor(FLIGHT_GRADES, device=DEV)[3 * sub[1] + sub[0], (4 * u[0]).long().clamp(max=3)]
    pos = [c.double() - 1 for c in chip]
    if case["pixadj"] == "RANDOMIZE":
        pos = [pos[0].floor() + u[1], pos[1].floor() + u[2]]
    elif case["pixadj"] != "EXACT":
        pos = [q.floor() + 0.5 for q in pos]
    if case["pixadj"] == "EDSER":
        rows, tab = T["acis/subpix_fi/rows"].cpu().numpy(), T["acis/subpix_fi/table"]
        last = {fg: (r, m) for r, (fg, m) in enumerate(rows.tolist())}     # a later row replaces an earlier one
        for fg, (r, m) in last.items():
            i = (grade == fg).nonzero().squeeze(1)
            if m <= 0 or not i.numel():
                continue
            e = tab[0, r, :m].contiguous()
            j = torch.searchsorted(e, ev["b_energy"][i]).clamp(1, m - 1)
            w1 = (ev["b_energy"][i].double() - e[j - 1].double()) / (e[j] - e[j - 1]).double()
            for c in range(2):
                t = tab[1 + c, r].double()
                pos[c][i] += ((1 - w1) * t[j - 1] + w1 * t[j]).float().double()
    mnc = torch.zeros(3, n, device=DEV, dtype=torch.float64)
    for c, ll, xh, yh, xl, yl in _chips(T):
        i = (ev["ccd"] == c).nonzero().squeeze(1)
        ofs = torch.stack([torch.full_like(ll[0], -10070.0), ll[1], ll[2]])    # the corner's x is left out, as marx2fits does
        mnc[:, i] = ofs[:, None] + (xh * (xl / 1024))[:, None] * pos[0][i] + (yh * (yl / 1024))[:, None] * pos[1][i]
    mnc = _unit(mnc)
    scale = 0.492 * ARCSEC
    out = {c: None for c in ("expno", "fltgrade", "grade", "tdetx", "tdety")}
    out["chipx"], out["chipy"] = chip
    out["detx"], out["dety"] = 4096.5 - mnc[1] / (scale * mnc[0]), 4096.5 + mnc[2] / (scale * mnc[0])
    ny, nz = -torch.sin(dec), torch.cos(dec) * torch.sin(ra)
    d = 2 * torch.sin(0.5 * dec) ** 2 + torch.cos(dec) * 2 * torch.sin(0.5 * ra) ** 2
    b = (mnc[1] * ny + mnc[2] * nz) / (2 - d)
    x, y, z = (mnc[0] + (ny * mnc[2] - nz * mnc[1] - d * mnc[0]), mnc[1] + (b * ny + nz * mnc[0] - d * mnc[1]),
               mnc[2] + (b * nz - ny * mnc[0] - d * mnc[2]))
    y, z = torch.cos(roll) * y - torch.sin(roll) * z, torch.cos(roll) * z + torch.sin(roll) * y
    out["x"] = 4096.5 - torch.atan2(-y, -x) / scale
    out["y"] = 4096.5 - torch.atan2(z, torch.sqrt(x * x + y * y)) / scale
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "events":
        return _exact_events(case, seed)
    if kind == "gradient":
        return _exact_gradient(case, seed)
    if kind in ("trace", "fef", "host"):
        cfg, name = W.ALL[case["workload"]]().cfg, case["workload"]
        energy, p, time = _inputs(name, case["n"], seed)
        if kind != "fef" and name in ("plain_onaxis", "plain_scatter"):
            return _trace_plain(cfg, energy, p, time, seed)
        dith = torch.zeros(3, case["n"], device=DEV, dtype=torch.float64)
        for k in range(2):
            dith[k] = (cfg.dither_amp[k] * ARCSEC * torch.sin(2 * math.pi * time / cfg.dither_period[k] + cfg.dither_phase[k])).float()
        roll = math.fmod(math.radians(cfg.roll_nom), 2 * math.pi)
        dith[2] = float(np.float32(roll - 2 * math.pi if roll >= math.pi else roll))
        return {"dither_state": dith}
    return None
