"""Performance cases: what a user has the framework do, from the smallest
calls to the largest, each through a public entry point.

* ``forward``: ``WavePropagator.forward_modeling`` (modelling observed data,
  a quick look at a model).
* ``misfit``: ``WavePropagator.misfit_gradient``, the evaluation that every
  iteration of an inversion is made of (forward, L2 residual, gradient).
* ``autograd``: ``torchfwi.Fwi`` forward and backward, for users whose misfit
  is written in torch.
* ``lowpass``: ``fwi_tools.lowpass`` of trace planes, as the multiscale
  inversion filters its data before each misfit.

The sizes are those of the repository's own configurations (the 100 x 100,
200 x 400, 500 x 1000 and 1000 x 3000 surveys of its benchmark and tests),
with fewer steps or shots where the whole survey would take many seconds, and
generic ones between and beside them.  Models, wavelets and observed data are
made from the seed: layered models with a lens, Ricker sources, observed
sections of moved-out Ricker arrivals.

``exact`` restates the path in float64 torch (the propagator, the reference
scheme's adjoint and imaging, the reverse-time reconstruction, the exact
derivative by autograd step by step, the filter by FFT).
"""
import math

import numpy as np
import torch

from pyfwi_b200 import acquisition, fwi_tools
from pyfwi_b200.torchfwi import Fwi
from pyfwi_b200.wave_propagation import WavePropagator

FIELDS = ("vx", "vz", "taux", "tauz", "tauxz")
KEYS = {0: ("taux", "tauz"), 1: ("taux",), 2: ("vx", "vz"), 3: ("taux", "tauz", "tauxz"), 4: FIELDS}
# device memory each survey's checkpoints may plan for: several surveys (or
# the rest of a user's program) share the card
MEMORY = 40e9
# the most cell-steps (cells x shots x steps) of a drawn survey
MOST_CELL_STEPS = 3.5e9

SURVEY = dict(kind="misfit", nz=100, nx=100, npml=20, dh=5.0, dt=0.0005, nt=500, ns=4, f0=10.0, order=4, components=2,
              acq=1, wells=0, rec_step=1, chpr=100, energy=False, param="dv", adjoint="reference", snapshot="fp32",
              water=0, host=False)


def _survey(**kw):
    return dict(SURVEY, **kw)


def listed():
    return [
        # a test-sized survey from numpy arrays: what a call costs at the least
        _survey(name="smallest_forward", kind="forward", nz=32, nx=40, npml=5, dh=2.0, dt=0.0004, nt=150, ns=2, f0=40.0,
                components=4, host=True),
        # the 100 x 100 survey of the reference's examples, whole: one evaluation of a small inversion
        _survey(name="small_gradient", nz=100, nx=100, npml=20, dh=1.0, dt=0.0002, nt=500, ns=4, f0=60.0),
        # the 200 x 400 survey: modelling its data, and an evaluation (half its record)
        _survey(name="medium_forward", kind="forward", nz=200, nx=400, npml=20, nt=1000, ns=10, components=0),
        _survey(name="medium_gradient", nz=200, nx=400, npml=20, nt=1000, ns=10, components=0),
        # the 500 x 1000 survey of the benchmark, a quarter of its shots and the first part of its record
        _survey(name="large_gradient", nz=500, nx=1000, npml=30, nt=600, ns=16, f0=8.0, components=0),
        # the thrust-belt grid with a water layer, two shots and the start of the record
        _survey(name="thrust_belt_gradient", nz=1000, nx=3000, npml=40, dh=4.0, dt=0.0004, nt=400, ns=2, f0=10.0,
                components=0, water=20),
        # a torch program: misfit in torch, gradient of the modelled section by autograd
        _survey(name="autograd_gradient", kind="autograd", nz=161, nx=301, npml=20, nt=600, ns=6, components=0),
        # the same with the exact derivative instead of the reference's gradient
        _survey(name="autograd_exact", kind="autograd", nz=101, nx=203, npml=20, nt=300, ns=4, components=0,
                adjoint="exact"),
        # eighth-order stencils, all components, energy-balanced lam / mu / rho gradient
        _survey(name="eighth_order_energy", nz=100, nx=150, npml=20, nt=900, ns=4, order=8, components=4, energy=True,
                param="lmd"),
        # the reference's low-memory scheme: one state in ten kept, the rest reconstructed in reverse time
        _survey(name="reconstructed_gradient", nz=150, nx=250, npml=20, nt=500, ns=5, components=3, chpr=10),
        # a coarse time sample that is sub-stepped, surface line and two wells
        _survey(name="substepped_wells", nz=140, nx=180, npml=15, dh=10.0, dt=0.0011, nt=260, ns=3, f0=8.0, components=4,
                acq=2, wells=60),
        # the multiscale filter on the 200 x 400 survey's two recorded planes
        dict(name="lowpass_traces", kind="lowpass", planes=2, nt=2000, traces=4000, dt=0.0005, highcut=15.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.08:
        return dict(kind="lowpass", planes=rng.choice((1, 2, 3, 5)), nt=_log(rng, 150, 4000),
                    traces=_log(rng, 60, 8000), dt=0.0005, highcut=rng.choice((5.0, 10.0, 15.0, 25.0)))
    c = _survey(kind=rng.choice(("misfit", "misfit", "misfit", "forward", "autograd")))
    c["nz"] = _log(rng, 30, 1000)
    c["nx"] = min(3000, max(40, int(c["nz"] * math.exp(rng.uniform(0.0, math.log(3.5))))))
    c["npml"] = rng.choice((8, 10, 15, 20, 30)) if c["nz"] >= 80 else 5
    c["ns"] = _log(rng, 1, 32)
    c["nt"] = _log(rng, 120, 1500)
    c["dh"], c["dt"], c["f0"] = rng.choice(((1.0, 0.0002, 60.0), (2.0, 0.0004, 40.0), (5.0, 0.0005, 10.0),
                                            (10.0, 0.0011, 8.0)))
    c["components"] = 0 if c["kind"] == "autograd" else rng.choice((0, 0, 2, 2, 1, 3, 4))
    c["rec_step"] = rng.choice((1, 1, 1, 2))
    if c["kind"] != "forward":
        option = rng.random()
        if option < 0.12:
            c["chpr"] = rng.choice((5, 10, 20))
        elif option < 0.20 and c["kind"] == "misfit":
            c["energy"], c["param"] = True, "lmd"
        elif option < 0.28:
            c["snapshot"] = "fp24"
        elif option < 0.33 and c["kind"] == "autograd":
            c["adjoint"] = "exact"
    if rng.random() < 0.12:
        c["order"] = 8
    if rng.random() < 0.1 and c["nz"] >= 80:
        c["water"] = rng.choice((6, 10, 20))
    if c["dt"] > 0.0006:
        c["nt"] = max(60, c["nt"] // 2)
    if c["energy"]:  # long enough to light every cell: the balancing divides by what arrived there
        c["nz"], c["nx"] = min(c["nz"], 120), min(c["nx"], 200)
        c["nt"] = max(c["nt"], int((2.0 / c["f0"] + 1.6 * c["nz"] * c["dh"] / 1500.0) / c["dt"]))
        c["ns"] = min(16, max(c["ns"], 4))
    if c["water"] and c["nt"] * c["dt"] < c["water"] * c["dh"] / 1500.0 + 1.0 / c["f0"]:
        c["water"] = 0  # nothing would reach the solid
    steps = math.ceil(c["dt"] / 0.0006)
    cost = (c["nz"] + 2 * c["npml"]) * (c["nx"] + 2 * c["npml"]) * c["ns"] * c["nt"] * steps
    if c["chpr"] != 100 or c["adjoint"] == "exact" or c["energy"] or c["order"] == 8:
        cost *= 2
    while cost > MOST_CELL_STEPS:
        f = min(0.75, max(0.25, MOST_CELL_STEPS / cost))
        k = "nt" if c["nt"] > 120 and not c["energy"] else "ns" if c["ns"] > 1 else "nx"
        old, c[k] = c[k], max(1, int(c[k] * f))
        cost *= c[k] / old
    c["host"] = c["kind"] == "forward" and c["nz"] < 120 and rng.random() < 0.5
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _model(c, rng):
    """vp, vs, rho (nz, nx) float32: layers and a lens, an optional water layer."""
    nz, nx = c["nz"], c["nx"]
    z, x = np.linspace(0, 1, nz)[:, None], np.linspace(0, 1, nx)[None, :]
    top = min(3900.0, 0.45 * c["dh"] / (c["dt"] / math.ceil(c["dt"] / 0.0006)))  # inside the stable time step
    lo, hi = min(1700.0, 0.75 * top), 0.9 * top
    vp = lo + (hi - lo) * z + 0 * x
    for _ in range(3):
        z0, slope, jump = rng.uniform(0.2, 0.85), rng.uniform(-0.15, 0.15), rng.uniform(-120.0, 180.0)
        vp = vp + jump / (1 + np.exp(-np.clip((z - z0 - slope * (x - 0.5)) * 0.5 * nz, -40, 40)))
    cz, cx, r = rng.uniform(0.35, 0.7), rng.uniform(0.25, 0.75), rng.uniform(0.08, 0.18)
    vp = np.clip(vp * (1 - 0.06 * np.exp(-(((z - cz) / r) ** 2 + ((x - cx) / r) ** 2))), 1200.0, top)
    vs, rho = vp / 1.8, 310 * vp ** 0.25
    if c["water"]:
        vp[:c["water"]], vs[:c["water"]], rho[:c["water"]] = 1500.0, 0.0, 1000.0
    return {k: v.astype(np.float32) for k, v in (("vp", vp), ("vs", vs), ("rho", rho))}


def _locations(c):
    """(src_loc, rec_loc) in metres, columns x then z."""
    nz, nx, dh, ns = c["nz"], c["nx"], c["dh"], c["ns"]
    src = np.stack([np.linspace(min(6, nx // 4), nx - 1 - min(6, nx // 4), ns).astype(np.int32) * dh,
                    np.full(ns, 2 * dh)], 1)
    xs = np.arange(1, nx - 1, c["rec_step"])
    rec = np.stack([xs * dh, np.full(xs.size, 2 * dh)], 1)
    if c["acq"] == 2:
        zs = 4 + np.arange(c["wells"])
        left = np.stack([np.full(zs.size, 3 * dh), zs * dh], 1)
        right = np.stack([np.full(zs.size, (nx - 4) * dh), zs * dh], 1)
        rec = np.vstack([left, rec, right])
    return src.astype(np.float32), rec.astype(np.float32)


def _inpa(c):
    inpa = {"dt": c["dt"], "t": (c["nt"] - 1) * c["dt"] + c["dt"] / 2, "dh": c["dh"], "npml": c["npml"], "pmlR": 1e-5,
            "pml_dir": 2, "sdo": c["order"], "rec_dis": c["dh"] * c["rec_step"], "acq_type": c["acq"]}
    if c["energy"]:
        inpa["energy_balancing"] = True
    if c["adjoint"] != "reference":
        inpa["adjoint"] = c["adjoint"]
    if c["snapshot"] != "fp32" and c["chpr"] == 100:
        inpa["snapshot"] = c["snapshot"]
    return inpa


def _ricker(t, f):
    a = (math.pi * f * t) ** 2
    return (1 - 2 * a) * torch.exp(-a)


def _observed(c, rng, dev):
    """An observed section: moved-out Ricker arrivals, (nt, ns * nr) float32 per key."""
    src, rec = _locations(c)
    off = np.abs(rec[None, :, 0] - src[:, None, 0]).reshape(-1)
    off = torch.from_numpy(off.astype(np.float32)).to(dev)
    t = (torch.arange(c["nt"], device=dev, dtype=torch.float32) * c["dt"] - 1.0 / c["f0"])[:, None]
    depth = c["nz"] * c["dh"]
    data = {}
    for k in KEYS[c["components"]]:
        a = torch.zeros((c["nt"], off.numel()), dtype=torch.float32, device=dev)
        for _ in range(3):
            v, h, amp = rng.uniform(1600.0, 2600.0), rng.uniform(0.0, 0.9) * depth, rng.uniform(0.005, 0.03)
            a += amp * _ricker(t - torch.sqrt(off * off + h * h)[None, :] / v, c["f0"])
        data[k] = a
    return data


def _inputs(c, seed, dev):
    rng = np.random.default_rng(seed)
    model = _model(c, rng)
    return model, (_observed(c, rng, dev) if c["kind"] != "forward" else None)


def _traces(c, seed, dev):
    g = torch.Generator(device="cpu").manual_seed(int(seed))
    x = torch.randn((c["planes"], c["nt"], c["traces"]), generator=g, dtype=torch.float32)
    return x.to(dev)


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def prepare(case, seed):
    c = case
    dev = _device()
    if c["kind"] == "lowpass":
        return {"case": c, "x": _traces(c, seed, dev), "fn": 1.0 / (2 * c["dt"])}
    model, obs = _inputs(c, seed, dev)
    src_loc, rec_loc = _locations(c)
    src = acquisition.Source(src_loc, c["dh"], c["dt"], 0)
    src.Ricker(c["f0"])
    W = WavePropagator(_inpa(c), src, rec_loc, (c["nz"], c["nx"]), components=c["components"],
                       n_well_rec=c["wells"], chpr=c["chpr"])
    W.memory_budget = MEMORY
    W.plan  # the device plan, built before the first call
    if not c["host"]:
        model = {k: torch.from_numpy(v).to(dev) for k, v in model.items()}
    return {"case": c, "W": W, "model": model, "obs": obs}


def run(state):
    c = state["case"]
    if c["kind"] == "lowpass":
        return fwi_tools.lowpass(state["x"], c["highcut"], state["fn"], order=1, axis=1)
    W, model, obs = state["W"], state["model"], state["obs"]
    if c["kind"] == "forward":
        return W.forward_modeling(model)
    if c["kind"] == "misfit":
        rms, grad = W.misfit_gradient(model, obs, parameterization=c["param"])
        return {"rms": rms, "grad": grad}
    leaves = {k: v.clone().requires_grad_(True) for k, v in model.items()}
    tx, tz = Fwi.apply(W, leaves["vp"], leaves["vs"], leaves["rho"])
    loss = 0.5 * ((tx - obs["taux"]) ** 2).sum() + 0.5 * ((tz - obs["tauz"]) ** 2).sum()
    loss.backward()
    return {"taux": tx.detach(), "tauz": tz.detach(), "grad": {k: v.grad for k, v in leaves.items()}}


# floating-point operations per cell and step, counted from the update
# formulas: a difference costs 5 (4th order) or 11 (8th order); a forward step
# has 8 differences and 40 further operations, an adjoint step with imaging 10
# differences and 70 (the imaged differences of the forward state counted with
# the forward step: two more)
def work(case):
    c = case
    if c["kind"] == "lowpass":
        n = c["planes"] * c["traces"]
        points = 2 ** math.ceil(math.log2(2 * c["nt"]))
        return {"bytes": 8 * n * c["nt"], "flops": 2 * 2.5 * n * points * math.log2(points)}
    diff = 5 if c["order"] == 4 else 11
    cells = (c["nz"] + 2 * c["npml"]) * (c["nx"] + 2 * c["npml"])
    steps = cells * c["ns"] * c["nt"] * math.ceil(c["dt"] / 0.0006)
    _, rec = _locations(c)
    section = 4 * len(KEYS[c["components"]]) * c["nt"] * c["ns"] * len(rec)
    model = 12 * c["nz"] * c["nx"]
    if c["kind"] == "forward":
        return {"bytes": model + section, "flops": steps * (8 * diff + 40)}
    return {"bytes": 2 * model + section * (3 if c["kind"] == "autograd" else 1),
            "flops": steps * (20 * diff + 112)}


# ---------------------------------------------------------------------------
# the same in float64
# ---------------------------------------------------------------------------
PAD = 4


class _Propagator64:
    """The propagator of one survey in float64 torch: fields (ns, tnz + 2 PAD,
    tnx + 2 PAD) with a zero frame, updates on rows / columns R .. N - R."""

    def __init__(self, c, model, dev):
        self.c, self.dev = c, dev
        self.R, self.npml = R, npml = c["order"] // 2, c["npml"]
        self.tnz, self.tnx = c["nz"] + 2 * npml, c["nx"] + 2 * npml
        r6 = lambda v: float("%f" % v)  # the reference's kernels see these rounded to six decimals
        self.scale = int(math.ceil(c["dt"] / 0.0006))
        dt = c["dt"] / self.scale
        t = (c["nt"] - 1) * c["dt"] + c["dt"] / 2
        self.nt, self.nt_ext = int(1 + t // dt), int(1 + t // c["dt"])
        self.dt = r6(dt)
        coef = (9 / 8, -1 / 24) if R == 2 else (1715 / 1434, -114 / 1434, 14 / 1434, -1 / 1434)
        self.coef = [r6(v) / r6(c["dh"]) for v in coef]
        zi = np.clip(np.arange(self.tnz) - npml, 0, c["nz"] - 1)
        xi = np.clip(np.arange(self.tnx) - npml, 0, c["nx"] - 1)
        self.zi, self.xi = torch.from_numpy(zi).to(dev), torch.from_numpy(xi).to(dev)
        m = {k: torch.from_numpy(v).to(dev, torch.float64) for k, v in model.items()}
        self.set_model(m)
        length = npml * np.float32(c["dh"])
        ramp = np.float32(-(3 / (2 * length)) * (((np.arange(npml) * np.float32(c["dh"])) / length) ** 2) * np.log10(1e-5))
        vmax = float(m["vp"].max())
        d = []
        for n in (self.tnz, self.tnx):
            a = np.zeros(n)
            a[n - npml:] = ramp
            a[:npml] = ramp[::-1]
            d.append(torch.from_numpy(a * vmax).to(dev))
        self.dz, self.dx = d[0][:, None].expand(self.tnz, self.tnx), d[1][None, :].expand(self.tnz, self.tnx)
        src, rec = _locations(c)
        dh = c["dh"]
        self.sj = torch.from_numpy(np.int64(src[:, 0] / dh) + npml + PAD).to(dev)
        self.si = torch.from_numpy(np.int64(src[:, 1] / dh) + npml + PAD).to(dev)
        self.rj = torch.from_numpy(np.int64(rec[:, 0] / dh) + npml + PAD).to(dev)
        self.ri = torch.from_numpy(np.int64(rec[:, 1] / dh) + npml + PAD).to(dev)
        self.cts = int(src[0, 1] / dh)
        f = c["f0"]
        tw = np.arange(-1.0 / f, 1.0 / f + c["dt"] / 3, c["dt"])
        self.w = np.float32((1.0 - 2.0 * (np.pi * f * tw) ** 2) * np.exp(-(np.pi * f * tw) ** 2)).astype(np.float64)
        self.lo, self.zhi, self.xhi = R, self.tnz - R, self.tnx - R

    def set_model(self, m):
        e = {k: v[self.zi][:, self.xi] for k, v in m.items()}
        self.mu = e["rho"] * e["vs"] ** 2
        self.lam = e["rho"] * e["vp"] ** 2 - 2 * self.mu
        self.b, self.rho = 1 / e["rho"], e["rho"]

    def zeros(self, ns):
        return [torch.zeros((ns, self.tnz + 2 * PAD, self.tnx + 2 * PAD), dtype=torch.float64, device=self.dev)
                for _ in range(5)]

    def padded(self, a):
        return torch.nn.functional.pad(a, (PAD, PAD, PAD, PAD))

    def at(self, f, box, dz=0, dx=0):
        r0, r1, c0, c1 = box
        return f[..., PAD + r0 + dz:PAD + r1 + 1 + dz, PAD + c0 + dx:PAD + c1 + 1 + dx]

    def box(self, inset=0):
        return (self.lo + inset, self.zhi - inset, self.lo + inset, self.xhi - inset)

    def d(self, f, box, axis, forward):
        o = 0
        for q, ck in enumerate(self.coef):
            hi, lo = (q + 1, -q) if forward else (q, -q - 1)
            a = self.at(f, box, hi, 0) if axis == "z" else self.at(f, box, 0, hi)
            b = self.at(f, box, lo, 0) if axis == "z" else self.at(f, box, 0, lo)
            o = o + ck * (a - b)
        return o

    def crop(self, a, box):
        return a[box[0]:box[1] + 1, box[2]:box[3] + 1]

    def velocity(self, S):
        """The increments b (D tau) of vx and vz on the update domain."""
        D = self.box()
        b = self.crop(self.b, D)
        return (b * (self.d(S[2], D, "x", False) + self.d(S[4], D, "z", False)),
                b * (self.d(S[3], D, "z", True) + self.d(S[4], D, "x", True)))

    def stress(self, S):
        D = self.box()
        lam, mu = self.crop(self.lam, D), self.crop(self.mu, D)
        ex, ez = self.d(S[0], D, "x", True), self.d(S[1], D, "z", False)
        return ((lam + 2 * mu) * ex + lam * ez, (lam + 2 * mu) * ez + lam * ex,
                mu * (self.d(S[1], D, "x", False) + self.d(S[0], D, "z", True)))

    def forward_step(self, S):
        D = self.box()
        g = 1 - self.dt * self.crop(self.dx + self.dz, D)
        for f, inc in zip((0, 1), self.velocity(S)):
            v = self.at(S[f], D)
            v += self.dt * inc
            v *= g
        for f, inc in zip((2, 3, 4), self.stress(S)):
            v = self.at(S[f], D)
            v += self.dt * inc
            v *= g

    def reverse_step(self, S):
        D = self.box()
        g = 1 - self.dt * self.crop(self.dx + self.dz, D)
        for f, inc in zip((2, 3, 4), self.stress(S)):
            v = self.at(S[f], D)
            v *= g
            v -= self.dt * inc
        for f, inc in zip((0, 1), self.velocity(S)):
            v = self.at(S[f], D)
            v *= g
            v -= self.dt * inc

    def sample(self, t):
        k = t // self.scale
        return self.w[k] if t % self.scale == 0 and k < self.w.size else 0.0

    def add_source(self, S, t, shots):
        w = self.sample(t)
        if w:
            i, j = self.si[shots], self.sj[shots]
            n = torch.arange(len(i), device=self.dev)
            S[2][n, i, j] += w
            S[3][n, i, j] += w

    def forward(self, shots, store=None):
        """Traces [5, nt_ext, ns, nr]; store[t] is called with the state after step t."""
        ns = len(self.si[shots])
        S = self.zeros(ns)
        tr = torch.zeros((5, self.nt_ext, ns, len(self.ri)), dtype=torch.float64, device=self.dev)
        for t in range(self.nt):
            if t % self.scale == 0:
                k = t // self.scale
                if k < self.nt_ext:
                    for f in range(5):
                        tr[f, k] = S[f][:, self.ri, self.rj]
                self.add_source(S, t, shots)
            self.forward_step(S)
            if store is not None:
                store(t, S)
        return tr

    def section(self, tr):
        """{key: (nt_ext, ns, nr)} of the case's components."""
        c = self.c
        if c["acq"] == 2:
            tr = tr.clone()
            tr[..., :c["wells"]] = tr[..., :c["wells"]].flip(-1)
        if c["components"] == 0:
            m = (tr[2] + tr[3]) / 2
            return {"taux": m, "tauz": m}
        return {k: tr[FIELDS.index(k)] for k in KEYS[c["components"]]}

    def inject(self, A, res, row):
        for k, r in res.items():
            f = A[FIELDS.index(k)]
            n = torch.arange(f.shape[0], device=self.dev)[:, None].expand(-1, len(self.ri))
            f.index_put_((n, self.ri[None].expand(f.shape[0], -1), self.rj[None].expand(f.shape[0], -1)), r[row],
                         accumulate=True)

    def adjoint_step(self, A):
        D = self.box()
        dx, dz, b = self.crop(self.dx, D), self.crop(self.dz, D), self.padded(self.b)
        lam, mu = self.padded(self.lam), self.padded(self.mu)
        bx, bz = b * A[0], b * A[1]
        tx, tz, txz = (self.at(A[f], D) for f in (2, 3, 4))
        tx -= self.dt * (dx * tx + self.d(bx, D, "x", True))
        tz -= self.dt * (dz * tz + self.d(bz, D, "z", False))
        txz -= self.dt * ((dx + dz) * txz + self.d(bx, D, "z", True) + self.d(bz, D, "x", False))
        pxx = (lam + 2 * mu) * A[2] + lam * A[3]
        pzz = (lam + 2 * mu) * A[3] + lam * A[2]
        pxz = mu * A[4]
        vx, vz = self.at(A[0], D), self.at(A[1], D)
        vx -= self.dt * ((2 * dx + dz) * vx + self.d(pxx, D, "x", False) + self.d(pxz, D, "z", False))
        vz -= self.dt * ((dx + 2 * dz) * vz + self.d(pzz, D, "z", True) + self.d(pxz, D, "x", True))

    def image(self, S, A, G):
        I = self.box(self.npml)
        dt = self.dt
        at = lambda F, f: self.at(F[f], I)
        b = self.crop(self.b, I)
        ex, ez = self.d(S[0], I, "x", True), self.d(S[1], I, "z", False)
        # the reference forms its "Dz+ vx" from vz
        sz, sx = self.d(S[1], I, "z", True), self.d(S[1], I, "x", False)
        pz, pxz_z = self.d(S[3], I, "z", True), self.d(S[4], I, "z", False)
        px, pxz_x = self.d(S[2], I, "x", False), self.d(S[4], I, "x", True)
        G[0] += (2 * dt * (at(A, 2) * ex + at(A, 3) * ez) + dt * at(A, 4) * (sz + sx)).sum(0)
        G[1] += (dt * (at(A, 2) + at(A, 3)) * (ex + ez)).sum(0)
        G[2] -= (dt * b * b * (at(A, 0) * (px + pxz_z) + at(A, 1) * (pz + pxz_x))).sum(0)
        if len(G) == 6:
            G[3] += (4 * dt * dt * (at(S, 2) ** 2 * ex ** 2 + at(S, 3) ** 2 * ez ** 2)
                     + dt * dt * at(S, 4) ** 2 * (sz ** 2 + sx ** 2)).sum(0)
            G[4] += (dt * dt * (at(S, 2) ** 2 + at(S, 3) ** 2) * (ex ** 2 + ez ** 2)).sum(0)
            G[5] += (dt * dt * (at(S, 0) ** 2 * (px ** 2 + pxz_z ** 2) + at(S, 1) ** 2 * (pz ** 2 + pxz_x ** 2))).sum(0)

    def gradient(self, shots, res, states, G, chp=None):
        """Adds the shots' imaging to G; states[t]: S after step t (None: reconstructed from the next)."""
        A = self.zeros(len(self.si[shots]))
        row, S = self.nt_ext, None
        for t in range(self.nt - 1, 0, -1):
            if chp is None or t in chp:
                S = [f.clone() for f in states[t]] if chp is not None else states[t]
            else:
                self.reverse_step(S)
            if t % self.scale == 0:
                row -= 1
                self.inject(A, res, row)
            self.adjoint_step(A)
            self.image(S, A, G)

    def read(self, G):
        """Mask, normalise and convert the accumulators as gradient_reading does."""
        c, R, n = self.c, self.R, self.npml
        I = self.box(n)
        full = []
        for g in G:
            a = torch.zeros((self.tnz, self.tnx), dtype=torch.float64, device=self.dev)
            self.crop(a, I).copy_(g)
            full.append(a[n:self.tnz - n, n:self.tnx - n])
        mask = torch.zeros((c["nz"], c["nx"]), dtype=torch.float64, device=self.dev)
        win = (slice(R + self.cts + 2, -R), slice(R, -R))
        mask[win] = 1
        out = []
        for q in range(3):
            f = mask
            if c["energy"]:
                f = torch.zeros_like(mask)
                f[win] = 1 / torch.sqrt(full[3 + q][win])
                f = f / f.abs().max()
            out.append(full[q] * f)
        gmu, glam, grho = out
        if c["param"] == "lmd":
            return {"lam": glam, "mu": gmu, "rho": grho}
        crop = lambda a: a[n:self.tnz - n, n:self.tnx - n]
        lam, mu, rho = crop(self.lam), crop(self.mu), crop(self.rho)
        vp, vs = torch.sqrt((lam + 2 * mu) / rho), torch.sqrt(mu / rho)
        return {"vp": 2 * vp * rho * glam, "vs": -4 * rho * vs * glam + 2 * vs * rho * gmu,
                "rho": glam * (vp ** 2 - 2 * vs ** 2) + gmu * vs ** 2 + grho}

    # ---- exact derivative, one step at a time through autograd ----
    def exact_gradient(self, shots, res, states, model):
        mats = [a.detach().clone().requires_grad_(True) for a in (self.lam, self.mu, self.b)]
        kept = self.lam, self.mu, self.b
        total = [torch.zeros_like(a) for a in mats]
        D = self.box()
        g = 1 - self.dt * self.crop(self.dx + self.dz, D)
        frame = (PAD + D[2], self.tnx + PAD - 1 - D[3], PAD + D[0], self.tnz + PAD - 1 - D[1])
        L = self.zeros(len(self.si[shots]))
        # components 0: both keys hold (txx + tzz) / 2
        half = (res["taux"] + res["tauz"]) / 2
        res = {"taux": half, "tauz": half}
        for t in range(self.nt - 1, -1, -1):
            S = [f.clone() for f in states[t - 1]] if t else self.zeros(L[0].shape[0])
            if t % self.scale == 0:
                self.add_source(S, t, shots)
            S = [f.requires_grad_(True) for f in S]
            self.lam, self.mu, self.b = mats
            put = lambda f, inc: torch.nn.functional.pad((self.at(f, D) + self.dt * inc) * g - self.at(f, D), frame) + f
            iv = self.velocity(S)
            N = [put(S[0], iv[0]), put(S[1], iv[1]), S[2], S[3], S[4]]
            it = self.stress(N)
            N = N[:2] + [put(S[2 + q], it[q]) for q in range(3)]
            out = torch.autograd.grad(N, S + mats, L)
            L = [a.detach().clone() for a in out[:5]]
            for a, q in zip(total, out[5:]):
                a += q
            if t % self.scale == 0 and t // self.scale < self.nt_ext:
                self.inject(L, res, t // self.scale)
        self.lam, self.mu, self.b = kept
        leaves = {k: torch.from_numpy(v).to(self.dev, torch.float64).requires_grad_(True) for k, v in model.items()}
        self.set_model(leaves)
        grads = torch.autograd.grad([self.lam, self.mu, self.b], list(leaves.values()), total)
        self.lam, self.mu, self.b = kept
        return dict(zip(leaves, grads))


def _lowpass64(c, x):
    n = c["nt"] + 512
    k = math.tan(math.pi * (2 * c["highcut"] * (2 * c["dt"])) / 2)  # first-order Butterworth by the bilinear transform
    z = torch.exp(2j * math.pi * torch.arange(n, dtype=torch.float64, device=x.device) / n)
    h = k * (z + 1) / ((z - 1) + k * (z + 1))
    X = torch.fft.fft(x.to(torch.float64), n=n, dim=1) * (h * h.conj()).real[None, :, None]
    return torch.fft.ifft(X, dim=1).real[:, :c["nt"]]


def exact(case, seed):
    c = case
    dev = _device()
    if c["kind"] == "lowpass":
        return _lowpass64(c, _traces(c, seed, dev))
    steps = math.ceil(c["dt"] / 0.0006) * c["nt"]
    cells = (c["nz"] + 2 * c["npml"] + 2 * PAD) * (c["nx"] + 2 * c["npml"] + 2 * PAD)
    # shots together: as many as keep their states (float64) within 45 GB
    kept = steps if c["chpr"] == 100 or c["kind"] == "forward" else max(2, c["chpr"] * steps // 100)
    batch = max(1, min(c["ns"], int(45e9 // (40.0 * cells * kept)) if c["kind"] != "forward" else c["ns"]))
    # about 70 (forward) and 200 (gradient) kernels a step, each some microseconds and its bytes
    ops = 70 if c["kind"] == "forward" else 500 if c["adjoint"] == "exact" else 200
    seconds = steps * ops * sum(7e-6 + 24.0 * cells * min(batch, c["ns"] - s) / 5e12 for s in range(0, c["ns"], batch))
    if seconds > 20 or 40.0 * cells * kept * batch > 60e9 and c["kind"] != "forward":
        return None
    model, obs = _inputs(c, seed, dev)
    P = _Propagator64(c, model, dev)
    parts, rms, G, grads = [], 0.0, None, None
    for s0 in range(0, c["ns"], batch):
        shots = slice(s0, min(s0 + batch, c["ns"]))
        if c["kind"] == "forward":
            parts.append(P.section(P.forward(shots)))
            continue
        chp = None
        if c["chpr"] != 100 and c["adjoint"] != "exact":
            chp = np.linspace(0, P.nt - 1, int(c["chpr"] * P.nt / 100), dtype=np.int32)
            chp = set((chp if len(chp) >= 2 else np.array([1, P.nt - 1])).tolist())
        states = {}

        def store(t, S):
            if chp is None or t in chp:
                states[t] = [f.clone() for f in S]

        sec = P.section(P.forward(shots, store))
        parts.append(sec)
        nr = len(P.ri)
        res = {k: v - obs[k].view(P.nt_ext, c["ns"], nr)[:, shots].to(torch.float64) for k, v in sec.items()}
        rms += sum(0.5 * float((r * r).sum()) for r in res.values())
        if c["adjoint"] == "exact":
            e = P.exact_gradient(shots, res, states, model)
            grads = e if grads is None else {k: grads[k] + e[k] for k in e}
        else:
            if G is None:
                I = P.box(P.npml)
                G = [torch.zeros((I[1] - I[0] + 1, I[3] - I[2] + 1), dtype=torch.float64, device=dev)
                     for _ in range(6 if c["energy"] else 3)]
            P.gradient(shots, res, states, G, chp)
        states.clear()
    section = {k: torch.cat([p[k] for p in parts], 1).reshape(P.nt_ext, -1) for k in parts[0]}
    if c["kind"] == "forward":
        return {k: v.cpu().numpy() for k, v in section.items()} if c["host"] else section
    grads = grads if grads is not None else P.read(G)
    if c["kind"] == "misfit":
        return {"rms": torch.tensor(rms, dtype=torch.float64), "grad": grads}
    return {"taux": section["taux"], "tauz": section["tauz"], "grad": grads}
