"""Timed workloads of the simulation path, through the package's public entry points.

A case is one piece of work that a program built on this package repeats: it
restores a simulation from a snapshot (crp_load_state), advances it, and reads
back the fields and bubble quantities it goes on with; or it asks for an
objective and its gradients (crp_adjoint); or it advances a batch of
simulations (crp_batch).  Grids, media, transducers and bubble populations are
those of cuda-rp_b200/configs and of the parity tests, and sizes between them.

listed()  the fixed cases; draw(rng) one more of the same ranges.
prepare() a simulation advanced to the start of the timed window, its snapshot
          and page-locked read-back buffers.
run()     one pass; it starts from the snapshot, so passes repeat.
work()    bytes and operations a pass cannot do without.
exact()   the same results from a plain 64-bit restatement of the model.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-rp_b200"))
import crp  # noqa: E402

RHO, C, P_INF = 998.0, 1482.0, 101325.0


def listed():
    return [
        # A few steps of the parity tests' 48 x 96 grid with the temperature
        # branch on (the reference's default): launches and host round trips.
        dict(name="small_48x96", kind="axisym", x=48, y=96, h=1e-4, pml=8, bubbles=500, amp=0.5e6, start=130, steps=10,
             precision="fp64", scheme="ref", temperature=True),
        # A save interval's share of the 256 x 512 configuration before the
        # burst reaches its 4,096 bubbles.
        dict(name="axisym_256x512", kind="axisym", x=256, y=512, h=1e-4, pml=16, bubbles=4096, amp=0.5e6, start=60,
             steps=40, precision="fp64", scheme="ref", temperature=False),
        # The 1024 x 2048 configuration (262,144 bubbles): the ordinary large
        # axisymmetric run, in both storage precisions.
        dict(name="axisym_1024x2048", kind="axisym", x=1024, y=2048, h=5e-5, pml=32, bubbles=262144, amp=2.0e6,
             start=60, steps=50, precision="fp64", scheme="ref", temperature=False),
        dict(name="axisym_1024x2048_mixed", kind="axisym", x=1024, y=2048, h=5e-5, pml=32, bubbles=262144, amp=2.0e6,
             start=60, steps=50, precision="mixed", scheme="ref", temperature=False),
        # The same grid once the burst drives the cloud: the stiffest bubble's
        # sub-steps set the time of every Picard iteration.
        dict(name="driven_1024x2048", kind="axisym", x=1024, y=2048, h=5e-5, pml=32, bubbles=262144, amp=2.0e6,
             start=1760, steps=5, precision="fp64", scheme="ref", temperature=False),
        # A driven cloud with the adaptive radius scheme.
        dict(name="driven_256x512_rk45", kind="axisym", x=256, y=512, h=1e-4, pml=16, bubbles=4096, amp=0.5e6,
             start=935, steps=20, precision="fp64", scheme="rk45", temperature=False),
        # Propagation without bubbles on a ragged grid with 64 source elements,
        # as a treatment-planning program runs it.
        dict(name="plain_1001x1531", kind="plain", x=1001, y=1531, h=1e-4, pml=20, elements=64, cylindrical=True,
             precision="fp64", start=20, steps=100),
        # Focal objective and its gradients over the elements, 2-D and 3-D:
        # one evaluation of an optimiser, forward and reverse.
        dict(name="adjoint_600x701", kind="adjoint2", x=600, y=701, h=1e-4, pml=16, elements=64, steps=300),
        dict(name="adjoint_141x125x133", kind="adjoint3", x=141, y=125, z=133, h=1.2e-4, pml=10, elements=64,
             steps=160),
        # The 256^3 configuration: 64 elements, 65,536 bubbles at the focus.
        dict(name="cart3d_256", kind="cart3d", x=256, y=256, z=256, h=1.2e-4, pml=24, elements=64, radius=100,
             bubbles=65536, cloud="sphere", sigma=16.7, r0=3e-6, sln=0.3, amp=1.0e6, freq=1.0e6, precision="fp64",
             start=10, steps=30),
        # The 384^3 configuration: 256 elements, 2,097,152 bubbles in a cloud
        # whose tail the burst already drives.
        dict(name="cart3d_384", kind="cart3d", x=384, y=384, z=384, h=1.0e-4, pml=24, elements=256, radius=160,
             bubbles=2097152, cloud="gaussian", sigma=30.0, r0=2e-6, sln=0.4, amp=1.0e6, freq=1.5e6, precision="fp64",
             start=25, steps=6),
        # A parameter sweep advanced as one batch.
        dict(name="sweep_16", kind="sweep", sims=16, layout=1, start=20, steps=40),
    ]


def draw(rng):
    def lg(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    kind = rng.choice(["axisym"] * 4 + ["plain"] * 2 + ["adjoint2", "adjoint3", "cart3d", "cart3d", "driven", "sweep"])
    if kind == "axisym":
        x = int(lg(48, 1000))
        y = max(96, min(2048, int(x * rng.uniform(1.3, 2.0))))
        cells = x * y
        bubbles = int(lg(64, min(250000, 0.08 * cells)))
        return dict(kind="axisym", x=x, y=y, h=rng.choice([5e-5, 1e-4]), pml=max(6, min(32, x // 16)), bubbles=bubbles,
                    amp=0.5e6, start=rng.randint(30, 60), steps=rng.randint(8, 50),
                    precision=rng.choice(["fp64", "fp64", "fp64", "mixed"]), scheme=rng.choice(["ref", "ref", "rk45"]),
                    temperature=rng.random() < 0.2)
    if kind == "plain":
        return dict(kind="plain", x=int(lg(64, 1400)), y=int(lg(96, 1400)), h=1e-4, pml=12,
                    elements=rng.randint(1, 96), cylindrical=rng.random() < 0.7,
                    precision=rng.choice(["fp64", "fp64", "mixed"]), start=rng.randint(5, 40),
                    steps=rng.randint(20, 120))
    if kind == "adjoint2":
        return dict(kind="adjoint2", x=int(lg(96, 640)), y=int(lg(128, 700)), h=1e-4, pml=12,
                    elements=rng.randint(2, 96), steps=rng.randint(150, 320))
    if kind == "adjoint3":
        return dict(kind="adjoint3", x=rng.randint(48, 140), y=rng.randint(48, 140), z=rng.randint(48, 140), h=1.2e-4,
                    pml=8, elements=rng.randint(4, 96), steps=rng.randint(90, 160))
    if kind == "cart3d":
        n = [int(lg(44, 230)) for _ in range(3)]
        r = min(n) / 2.0
        sigma = round(0.13 * r, 2)
        most = min(100000, int(6 * 4 / 3 * math.pi * sigma ** 3))  # a few bubbles per cell of the cloud
        return dict(kind="cart3d", x=n[0], y=n[1], z=n[2], h=1.2e-4, pml=8, elements=rng.randint(8, 128),
                    radius=round(r - 11.27, 2), bubbles=int(lg(64, most)), cloud=rng.choice(["sphere", "gaussian"]),
                    sigma=sigma, r0=3e-6, sln=0.3, amp=0.2e6, freq=1.0e6,
                    precision=rng.choice(["fp64", "fp64", "mixed"]), start=rng.randint(4, 10), steps=rng.randint(6, 20))
    if kind == "driven":
        return dict(kind="axisym", x=256, y=512, h=1e-4, pml=16, bubbles=int(lg(1000, 16000)), amp=0.5e6,
                    start=rng.randint(900, 940), steps=rng.randint(5, 20), precision="fp64",
                    scheme=rng.choice(["ref", "rk45"]), temperature=False)
    return dict(kind="sweep", sims=rng.randint(3, 16), layout=rng.randint(2, 10**6), start=rng.randint(5, 30),
                steps=rng.randint(10, 50))


# ---------------------------------------------------------------------------
# Configurations and seeded inputs.


def config(case, u):
    """The crp configuration of a case; u in [0, 1) shifts the drive by up to 5 %."""
    c = crp.defaults()
    c.grid_x, c.grid_y = case["x"], case["y"]
    c.grid_lx, c.grid_ly = case["x"] * case["h"], case["y"] * case["h"]
    c.pml_x0, c.pml_x1, c.pml_y0, c.pml_y1 = 0, 1, 1, 1
    c.pml_grid_number, c.pml_sigma, c.pml_order = case["pml"], 0.01, 2
    c.sim_cfl, c.sim_dt0, c.sim_order, c.sim_smooth_delta_band = 0.4, 0.1, 2, 2
    c.tr_freq, c.tr_on_wave, c.tr_off_wave = case.get("freq", 1.0e6), 20, 1000
    c.tr_amp = case.get("amp", 0.5e6) * (1.0 + 0.05 * u) / (RHO * C)
    c.ext_rho_inf, c.ext_c_inf, c.ext_p_inf, c.ext_ramp_cycles = RHO, C, P_INF, 3.0
    c.bub_R0, c.bub_P0, c.bub_T0, c.bub_gamma = 3e-6, P_INF, 293.15, 1.4
    c.bub_sigma, c.bub_mu, c.bub_rho, c.bub_K0 = 0.0725, 1e-3, RHO, 26.2e-3
    c.dbg_T = 1 if case.get("temperature") else 0
    c.bub_enable = 1 if case.get("bubbles") else 0
    c.ext_precision = 1 if case.get("precision") == "mixed" else 0
    if case.get("scheme") == "rk45":
        c.ext_rp_scheme, c.ext_rp_tol = 1, 1e-4
    if "z" in case:
        c.pml_x0 = c.ext_pml_z0 = c.ext_pml_z1 = 1
        c.ext_grid_z, c.ext_grid_lz = case["z"], case["z"] * case["h"]
        c.ext_array_elements = case["elements"]
        radius = case.get("radius", min(case["x"], case["y"], case["z"]) / 2.0 - case["pml"] - 3.27)
        c.ext_array_radius, c.ext_array_phases = radius * case["h"], 0
    else:
        c.tr_cylindrical = 1 if case.get("cylindrical", True) else 0
        c.tr_focused_p = 1
        c.ext_source_row = case["pml"] + 1
        c.ext_elements = case.get("elements", 0)
        # The focus: 34.6 mm deep on the two named grids, else at 60 % of the
        # length (40 % for the adjoint, whose steps have to reach it).
        depth = 0.40 * c.grid_ly if case["kind"] == "adjoint2" else 0.6 * c.grid_ly
        if case.get("bubbles") and (case["x"], case["y"]) in ((256, 512), (1024, 2048)):
            depth = 0.5 * math.sqrt(3.0) * 40e-3
        if case["kind"] == "adjoint2":
            depth = min(depth, (case["pml"] + 1 + 0.25 * case["steps"]) * case["h"])
        c.tr_focal_dist = depth * 2.0 / math.sqrt(3.0)
    return c


def focus(c):
    return c.tr_focal_dist * 0.5 * math.sqrt(3.0)


def population(case, c, rng):
    """Explicit bubbles: a cylinder about the axis at the focus (2-D), a ball
    or a Gaussian cloud about the centre (3-D); lognormal radii."""
    n = case["bubbles"]
    r0 = np.clip(case.get("r0", 3e-6) * np.exp(case.get("sln", 0.3) * rng.standard_normal(n)), 4e-7, 2e-5)
    one = np.ones(n)
    if "z" not in case:
        # 3 mm x 12 mm on the 1024 x 2048 grid, 2 mm x 8 mm on 256 x 512.
        rr, hh = {1024: (3e-3, 12e-3), 256: (2e-3, 8e-3)}.get(case["x"], (0.08 * c.grid_lx, 0.15 * c.grid_ly))
        x = rr * np.sqrt(rng.random(n))
        y = focus(c) + hh * (rng.random(n) - 0.5)
        return crp.Bubbles(np.maximum(x, 0.02 * case["h"]), y, r0, one)
    s = case["sigma"] * case["h"]
    ctr = [0.5 * case[k] * case["h"] for k in "xyz"]
    if case["cloud"] == "gaussian":
        v = s * rng.standard_normal((3, n))
    else:
        v = rng.standard_normal((3, n))
        v *= s * np.cbrt(rng.random(n)) / np.sqrt((v * v).sum(0))
    p = [np.ascontiguousarray(np.clip(ctr[k] + v[k], 2.5 * case["h"], 2 * ctr[k] - 2.5 * case["h"])) for k in range(3)]
    return crp.Bubbles(p[0], p[1], r0, one, p[2])


def inputs(case, seed):
    """Configuration, bubbles (or None) and source elements (or None)."""
    rng = np.random.default_rng(seed)
    c = config(case, float(rng.random()))
    bub = population(case, c, rng) if case.get("bubbles") else None
    elem = None
    if case.get("elements"):
        elem = 1.0 + 0.1 * rng.standard_normal(case["elements"]), 0.2 * rng.standard_normal(case["elements"])
    return c, bub, elem


def sweep_cases(case):
    """The simulations of a sweep, one case each: grids, drives and populations
    in the ranges of the benchmark's sweep."""
    r = random.Random(case["layout"])
    out = []
    for _ in range(case["sims"]):
        x = r.randint(128, 400) // 8 * 8
        out.append(dict(kind="axisym", x=x, y=2 * x, h=1e-4, pml=16, bubbles=int(math.exp(r.uniform(math.log(1e3),
                        math.log(3e4)))), amp=r.uniform(0.2e6, 1.0e6), freq=r.uniform(0.5e6, 2.0e6),
                        r0=r.uniform(2e-6, 5e-6), start=case["start"], steps=case["steps"], precision="fp64",
                        scheme="ref"))
    return out


# ---------------------------------------------------------------------------
# The pass.


def pinned(shape):
    t = torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    return t.numpy()


def outputs_of(case):
    if case["kind"] == "plain":
        return ["p0", "vx", "vy"], []
    if case["kind"] == "cart3d":
        return ["p0"], ["R_t", "PG_p", "x"]
    return ["p0", "vx", "vy", "f_g"] + (["T"] if case.get("temperature") else []), ["R_t", "PG_p", "x"]


def buffers(case, sim):
    fields, bubbles = outputs_of(case)
    shape = (lambda f: crp.field_shape3(sim.dims3, f)) if sim.dims3 is not None else (
        lambda f: crp.field_shape(sim.dims, f))
    return {f: pinned(shape(f)) for f in fields}, {b: pinned((sim.dims.num_bubbles if sim.dims3 is None else
                                                              sim.dims3.num_bubbles,)) for b in bubbles}


def read(sim, fields, bubbles):
    out = {}
    for f, buf in fields.items():
        out[f] = sim.field(f, buf)
    for b, buf in bubbles.items():
        out[b] = sim.bubbles(b, buf)
    return out


def focal_radius(case):
    return 8.3 * case["h"]


def prepare(case, seed):
    if case["kind"] == "sweep":
        parts = sweep_cases(case)
        made = [inputs(p, 1000 * seed + k) for k, p in enumerate(parts)]
        batch = crp.Batch([m[0] for m in made], [m[1] for m in made])
        batch.run([case["start"]] * len(parts))
        snaps = [s.save_state() for s in batch.sims]
        bufs = [({"p0": pinned(crp.field_shape(s.dims, "p0"))}, {"R_t": pinned((s.dims.num_bubbles,))})
                for s in batch.sims]
        return dict(case=case, batch=batch, snaps=snaps, bufs=bufs, steps=[case["steps"]] * len(parts), keep=made)
    c, bub, elem = inputs(case, seed)
    sim = crp.Sim(c, bub)
    if elem is not None:
        sim.set_source_elements(*elem)
    if case.get("start"):
        sim.step(case["start"])
    s = dict(case=case, sim=sim, snap=sim.save_state(), keep=(c, bub, elem))
    if case["kind"] not in ("adjoint2", "adjoint3"):
        s["bufs"] = buffers(case, sim)
    return s


def run(state):
    case = state["case"]
    if "batch" in state:
        for sim, snap in zip(state["batch"].sims, state["snaps"]):
            sim.load_state(snap)
        state["batch"].run(state["steps"])
        return [read(sim, *bufs) for sim, bufs in zip(state["batch"].sims, state["bufs"])]
    sim = state["sim"]
    sim.load_state(state["snap"])
    if case["kind"] in ("adjoint2", "adjoint3"):
        J, ga, gp = sim.adjoint(case["steps"], focal_radius(case), case["elements"])
        return {"J": J, "grad_amp": ga, "grad_phase": gp}
    sim.step(case["steps"])
    return read(sim, *state["bufs"])


def work(case):
    """Per step: velocities and split pressures read and written once (8 bytes
    each in both precisions), the void fraction not counted where no bubble
    is; about 20 operations per cell and dimension; per bubble its state read and
    written once and 10 sub-steps of about 300 operations.  The outputs are
    read back once.  The adjoint adds a reverse step that moves as much."""
    if case["kind"] == "sweep":
        w = [work(p) for p in sweep_cases(case)]
        return {k: sum(v[k] for v in w) for k in ("bytes", "flops")}
    dim = 3 if "z" in case else 2
    cells = case["x"] * case["y"] * case.get("z", 1)
    nb = case.get("bubbles", 0)
    per_step = cells * dim * 32 + nb * 200
    flops = cells * dim * 20 + nb * 10 * 300
    if case["kind"] in ("adjoint2", "adjoint3"):
        return {"bytes": 2.0 * per_step * case["steps"], "flops": 2.0 * flops * case["steps"]}
    fields, bubbles = outputs_of(case)
    out = 8 * (len(fields) * cells + len(bubbles) * nb)
    return {"bytes": float(per_step * case["steps"] + out), "flops": float(flops * case["steps"])}


# ---------------------------------------------------------------------------
# The model in plain 64-bit torch.


def _axis(n, npml, h, lo, hi, s4):
    """PML factors of one axis: faces 0..n (1 - s, 1 / (1 + s)), cells 1..n."""
    smax = -math.log(0.01) * 1.5 / (h * npml)
    face, cell = np.zeros(n + 1), np.zeros(n)
    f, k = np.arange(n + 1.0), np.arange(1.0, n + 1)
    if lo:
        face = np.where(f <= npml - 1, smax * ((npml - f) / npml) ** 2, face)
        cell = np.where(k <= npml, smax * ((npml - k + 0.5) / npml) ** 2, cell)
    if hi:
        face = np.where(f >= n - npml + 1, smax * ((f - n + npml) / npml) ** 2, face)
        cell = np.where(k >= n - npml + 1, smax * ((k - n + npml - 0.5) / npml) ** 2, cell)
    return 1 - s4 * face, 1 / (1 + s4 * face), 1 - s4 * cell, 1 / (1 + s4 * cell)


class _Model:
    """The bubbly-mixture model on a 2-D (axes y, x) or 3-D (axes z, y, x)
    staggered grid with a pressure source, as the package's configurations set
    it: per axis d, faces v[d] (n + 1 along d) and pressure parts p[d]."""

    def __init__(self, case, c, bub, elem, dev):
        self.dev, self.c, self.case = dev, c, case
        self.dim = 3 if "z" in case else 2
        self.n = [case[k] for k in ("zyx" if self.dim == 3 else "yx")]
        L = [c.ext_grid_lz, c.grid_ly, c.grid_lx][3 - self.dim:]
        self.h = [a / n for a, n in zip(L, self.n)]
        self.dt = c.sim_cfl * min(self.h) / C
        t = self.t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)
        z = lambda *s: torch.zeros(*s, dtype=torch.float64, device=dev)  # noqa: E731
        self.v = [z([n + (a == d) for a, n in enumerate(self.n)]) for d in range(self.dim)]
        self.p = [z(self.n) for _ in range(self.dim)]
        self.time = self.carry = 0.0
        self.first = True
        lo = [True] * self.dim
        if self.dim == 2:
            lo[1] = False
        self.fac = []
        for d in range(self.dim):
            s = [1] * self.dim
            s[d] = -1
            self.fac.append([t(f).reshape(s) for f in _axis(self.n[d], c.pml_grid_number, self.h[d], lo[d], True,
                                                             0.5 * self.dt * C)])
        self.cyl = self.dim == 2 and c.tr_cylindrical
        self.amp, self.phase = (None, None) if elem is None else (t(elem[0]), t(elem[1]))
        self.source_cells()
        self.fg = None
        if bub is not None:
            self.pos = [t(a) for a in ((bub.z, bub.y, bub.x) if self.dim == 3 else (bub.y, bub.x))]
            self.R0, self.nB = t(bub.r0), t(bub.n_b)
            self.Rt = self.Rp = self.Rn = self.R0.clone()
            o = torch.zeros_like(self.R0)
            self.d1, self.PLp, self.PLn, self.re = o, o.clone(), o.clone(), o.clone()
            self.PG = P_INF + 2 * c.bub_sigma / self.R0
            self.dtb = o + 0.1 * self.dt
            self.index()
            g = self.scatter(self.Rt)
            self.fg = [g, g.clone(), g.clone()]

    # Source ------------------------------------------------------------------
    def source_cells(self):
        c, case, t = self.c, self.case, self.t
        if self.dim == 2:
            x = (np.arange(1, self.n[1] + 1) - 0.5) * self.h[1]
            ym = (c.ext_source_row - 0.5) * self.h[0]
            cy = focus(c)
            self.fdist = cy / 0.5 / math.sqrt(3.0)
            s1 = np.sqrt(x * x + (cy - ym) ** 2)
            self.on = t(s1) <= self.fdist
            self.s1 = t(s1)
            if c.ext_elements:
                rap = np.abs(x)[s1 <= self.fdist].max()
                self.el = torch.as_tensor(np.minimum((np.abs(x) * c.ext_elements / rap).astype(np.int64),
                                                     c.ext_elements - 1), device=self.dev)
            return
        Ra, h = c.ext_array_radius, self.h
        ctr = [0.5 * n * a for n, a in zip(self.n, h)]
        e = np.arange(c.ext_array_elements)
        ct = -(e + 0.5) / c.ext_array_elements
        st = np.sqrt(1 - ct * ct)
        ph = math.pi * (3 - math.sqrt(5.0)) * e
        pts = np.stack([Ra * ct, Ra * st * np.sin(ph), Ra * st * np.cos(ph)], 1)
        q = [t((np.arange(1, n + 1) - 0.5) * a - m) for n, a, m in zip(self.n, h, ctr)]
        r = torch.sqrt(q[0].view(-1, 1, 1) ** 2 + q[1].view(1, -1, 1) ** 2 + q[2].view(1, 1, -1) ** 2)
        mask = ((r - Ra).abs() <= 0.5 * h[2]) & (q[0].view(-1, 1, 1) < 0)
        self.src = mask.nonzero(as_tuple=True)
        xyz = torch.stack([q[d][self.src[d]] for d in range(3)], 1)
        self.el = ((xyz[:, None, :] - t(pts)[None]) ** 2).sum(2).argmin(1)

    def envelope(self, tau):
        c = self.c
        ramp, rest = c.ext_ramp_cycles / c.tr_freq, c.tr_on_wave / c.tr_freq - tau
        up = 0.5 * (1 - torch.cos(math.pi * tau / ramp))
        down = torch.where(rest > 0, 0.5 * (1 - torch.cos(math.pi * rest / ramp)), torch.zeros_like(rest))
        w = torch.where(tau < ramp, up, torch.ones_like(tau))
        return torch.where(rest < ramp, torch.minimum(w, down), w)

    def source(self, time):
        c = self.c
        om, amp = 2 * math.pi * c.tr_freq, RHO * C * c.tr_amp
        on = c.tr_on_wave / c.tr_freq
        if self.dim == 2:
            tau = torch.clamp(time - (self.fdist - self.s1) / C, min=0.0)
            a, ph = (amp, 0.0) if self.amp is None else (amp * self.amp[self.el], self.phase[self.el])
            s = a * self.envelope(tau) * torch.sin(om * tau + ph)
            return torch.where(self.on & (tau < on), s, torch.zeros_like(s)) * (1.0 if time > 0 else 0.0)
        if not 0 < time <= on:
            return torch.zeros(len(self.el), dtype=torch.float64, device=self.dev)
        env = self.envelope(self.t(time))
        return (amp * self.amp * env * torch.sin(om * time + self.phase))[self.el]

    # Grid --------------------------------------------------------------------
    def p0(self, p, time):
        """Pressure with its source values and a ring of boundary cells."""
        q = sum(p[1:], p[0]) if self.dim == 2 else p[2] + p[1] + p[0]
        if self.dim == 2:
            row = torch.zeros(self.n[0], 1, dtype=torch.bool, device=self.dev)
            row[self.c.ext_source_row - 1] = True
            q = torch.where(row, self.source(time)[None], q)
            left = q[:, :1]
            q = torch.cat([left, q, torch.zeros_like(left)], 1)
            return torch.nn.functional.pad(q, (0, 0, 1, 1))
        return torch.nn.functional.pad(q, (1, 1) * 3)

    def diff(self, a, d):
        return a.narrow(d, 1, a.shape[d] - 1) - a.narrow(d, 0, a.shape[d] - 1)

    def inner(self, a, but):
        for d in range(self.dim):
            if d != but:
                a = a.narrow(d, 1, a.shape[d] - 2)
        return a

    def pressure(self, vn, fg, fgn):
        half = 0.0
        if fg is not None:
            a, b = self.inner(fg, -1), self.inner(fgn, -1)
            half = 0.5 * (-(a - b) / self.dt / (1 - 0.5 * (a + b)))
        out = []
        for d in range(self.dim):
            v = vn[d]
            if self.cyl and d == 1:
                i = self.t(np.arange(self.n[1] + 1.0)) * self.h[1]
                m = 1.0 / (self.h[1] * (self.t(np.arange(1.0, self.n[1] + 1)) - 0.5))
                s = self.diff(v * i, 1) / self.h[1] * m
            else:
                s = self.diff(v, d) / self.h[d]
            pa, pb = self.fac[d][2:]
            out.append(self.p[d] * pa - self.dt * RHO * C * C * (s + half) * pb)
        if self.dim == 3:
            f = self.source(self.time)
            z = torch.zeros_like(f)
            out = [o.index_put(self.src, f if d == 2 else z) for d, o in enumerate(out)]
        return out

    def step(self):
        t_prev = self.time
        t = t_prev + self.dt + self.carry
        self.carry = self.dt + self.carry - (t - t_prev)
        self.time = t
        p0 = self.p0(self.p, t_prev)
        fgp = None
        rho = None
        if self.fg is not None:
            a, b, g = self.fg
            fgp = 3 * a - 3 * b + g
            rho = torch.full_like(a, RHO) if self.first else (1 - a) * RHO
        vn = []
        for d in range(self.dim):
            va, vb = self.fac[d][:2]
            grad = self.diff(self.inner(p0, d), d) / (self.h[1] if self.dim == 2 else self.h[d])
            if rho is None:
                q = self.dt / RHO
            else:
                r = self.inner(rho, d)
                q = self.dt / (0.5 * (r.narrow(d, 0, r.shape[d] - 1) + r.narrow(d, 1, r.shape[d] - 1)))
            v = (self.v[d] * va - q * grad) * vb
            if self.dim == 2 and d == 1:
                v = torch.cat([torch.zeros_like(v[:, :1]), v[:, 1:]], 1)
            vn.append(v)
        pn = self.p
        new = self.pressure(vn, fgp, None if self.fg is None else self.fg[0])
        if self.fg is not None:
            self.move(vn)
            hist = self.fg
            self.fg = [fgp, hist[0], hist[1]]
            q0 = self.inner(self.p0(new, t), -1)
            res = (self.inner(p0, -1) - q0).abs().max().item() / P_INF
            tol = 1e-5 if self.c.ext_precision == 1 else float(np.float32(1e-7))
            start = self.begin_bubbles()
            while res > tol:
                Rt = self.radius(start, self.gather(self.p0(new, t)))
                self.fg[0] = self.scatter(Rt)
                self.p = pn
                nxt = self.pressure(vn, self.fg[0], hist[0])
                q1 = self.inner(self.p0(nxt, t), -1)
                res = (q0 - q1).abs().max().item() / P_INF
                new, q0 = nxt, q1
        self.p, self.v, self.first = new, vn, False

    # Bubbles -----------------------------------------------------------------
    def index(self):
        self.im = [torch.floor(x / h + 1.0).long() for x, h in zip(self.pos, self.h)]
        self.inn = [torch.floor(x / h + 0.5).long() for x, h in zip(self.pos, self.h)]

    def weight(self, d, pos, half=0.5):
        return 0.5 * (1 + torch.cos(math.pi / self.h[d] * ((pos.double() - 0.5) * self.h[d] - self.pos[d])))

    def stencil(self, a, base, off):
        """Sum of a over the bubbles' 2^dim points from `base`; off: index of point 0 per axis."""
        s = 0.0
        for k in range(1 << self.dim):
            ix, w = [], 1.0
            for d in range(self.dim):
                p = base[d] + ((k >> d) & 1)
                ix.append(p + off[d])
                w = w * self.weight(d, p)
            s = s + a[tuple(ix)] * w
        return s

    def gather(self, p0):
        return self.stencil(p0, self.inn, [0] * self.dim)

    def scatter(self, R):
        g = torch.zeros([n + 2 for n in self.n], dtype=torch.float64, device=self.dev)
        vol = math.pi * 4.0 / 3.0 * self.nB * R ** 3 / math.prod(self.h)
        if self.cyl:
            vol = vol / self.pos[1]
        for k in range(1 << self.dim):
            ix, w = [], vol
            for d in range(self.dim):
                p = self.inn[d] + ((k >> d) & 1)
                ix.append(p)
                w = w * self.weight(d, p)
            g.index_put_(tuple(ix), w, accumulate=True)
        if self.cyl:
            s = g[:, 0] + g[:, 1]
            g[:, 0] = s
            g[:, 1] = s
        return g

    def move(self, vn):
        vel = []
        for d in range(self.dim):
            v = vn[d]
            for e in range(self.dim):  # the boundary ring across the other axes
                if e == d:
                    continue
                if self.dim == 2 and e == 1:
                    v = torch.cat([v[:, :1], v, torch.zeros_like(v[:, :1])], 1)
                else:
                    v = torch.nn.functional.pad(v, [x for q in reversed(range(self.dim)) for x in
                                                    ((1, 1) if q == e else (0, 0))])
            off = [0] * self.dim
            if self.dim == 2 and d == 1:  # vx(-1) = vx(1)
                v = torch.cat([v[:, 1:2], v], 1)
                off[1] = 1
            base = [self.im[e] - 1 if e == d else self.inn[e] for e in range(self.dim)]
            vel.append(self.stencil(v, base, off))
        self.pos = [x + u * self.dt for x, u in zip(self.pos, vel)]
        self.index()

    def begin_bubbles(self):
        s = dict(Rt=self.Rt, Rp=self.Rp, Rn=self.Rn, d1=self.d1, PG=self.PG, PLn=self.PLp, PLm=self.PLn, dt=self.dtb,
                 re=self.re)
        self.PLn = self.PLp
        return s

    def thermal(self, PG, R):
        c = self.c
        PG0 = P_INF + 2 * c.bub_sigma / self.R0
        ca = c.bub_gamma * PG0 * self.R0 ** 3 / (2 * (c.bub_gamma - 1) * c.bub_T0 * c.bub_K0)
        c1 = PG0 / (PG * (R / self.R0) ** 3)
        eta = 3 * c.bub_gamma * c1 * PG * RHO - 2 * c.bub_sigma * RHO / R - 4 * c.bub_mu ** 2 / R ** 2
        floor = 1e-6 * 2.220446049250313e-16

        def omega(e):
            return torch.sqrt(torch.clamp(e, min=floor)) / (RHO * R)

        def coth_a(a):
            return a / torch.tanh(a) - 1

        om = omega(eta)
        for _ in range(3):
            s = torch.sqrt(ca * om / R)
            a = torch.complex(s, s)
            aa = torch.complex(torch.zeros_like(s), 2 * s * s)
            small = a.abs() <= 0.1
            t = torch.where(small, 1 / 3 + aa * (-1 / 45 + aa * (2 / 945 - aa / 4725)), coth_a(a) / aa)
            u = 3 * c.bub_gamma / (1 + 3 * (c.bub_gamma - 1) * t) * c1
            mu = c.bub_mu + u.imag * PG / (4 * om)
            eta = u.real * PG * RHO - 2 * c.bub_sigma * RHO / R - 4 * mu * mu / R ** 2
            om = omega(eta)
        s = torch.sqrt(ca * om / R)
        a = torch.complex(s, s)
        aa = torch.complex(torch.zeros_like(s), 2 * s * s)
        k = coth_a(a)
        lp = torch.where(a.abs() <= 0.1, 0.2 + aa * (-1 / 175 + aa * (2 / 7875 - 37 * aa / 3031875)),
                         (aa - 3 * k) / (aa * k)) * R
        return om, lp

    def radius(self, s, PLp):
        """All bubbles over one step with the three-level variable-step scheme."""
        c, dt = self.c, self.dt
        sg, mu, gam = c.bub_sigma, c.bub_mu, c.bub_gamma
        PLn, PLm = s["PLn"], s["PLm"]
        C0, C1, C2 = PLn + P_INF, 0.5 * (PLp - PLm) / dt, 0.5 * (PLp + PLm - 2 * PLn) / dt ** 2
        Rt, Rp, Rn, d1, PG, h = s["Rt"], s["Rp"], s["Rn"], s["d1"], s["PG"], s["dt"]
        rem, tm = s["re"] + dt, -s["re"]
        PG0 = P_INF + 2 * sg / self.R0
        eps = 2.220446049250313e-16
        for _ in range(400):
            on = rem > 0
            if not bool(on.any()):
                break
            R, m = Rp, Rn
            PL = C2 * tm * tm + C1 * tm + C0
            acc = (PG - PL - 2 * sg / R - 4 * mu / R * d1) / RHO - 1.5 * d1 * d1
            hp = torch.clamp(1.01 * h, max=0.1 * dt)
            hp = torch.where(d1.abs() > eps, torch.minimum(hp, 0.01 * R / d1.abs()), hp)
            hp = torch.where(acc.abs() > eps, torch.minimum(hp, 0.1 * R / torch.sqrt(acc.abs())), hp)
            q = hp / h
            nR = (1 + q) * R - q * m + hp / R * (0.5 * (hp + h) * acc)
            nd = (h * h * nR + (hp * hp - h * h) * R - hp * hp * m) / (h * hp * (h + hp)) + hp / R * acc
            last = hp >= rem
            step = torch.where(last, rem, hp)
            ql = step / h
            nt = torch.where(last, (1 + ql) * R - ql * m + step / R * (0.5 * (step + h) * acc), nR)
            om, lp = self.thermal(PG, R)
            den = lp.real ** 2 + lp.imag ** 2
            mid = 0.5 * (nR + R)
            c0 = hp * 3 * (gam - 1) * c.bub_K0 * c.bub_T0 / (mid * PG0)
            Lr, w = lp.real / den, c0 * lp.imag / den / (om * hp)
            c3 = c0 * Lr * 0.5 * (mid / self.R0) ** 3 + 1.5 * gam * (nR - R) / mid
            nPG = ((1 - c3 - w * (R / self.R0) ** 3) * PG + c0 * Lr * PG0) / (1 + c3 - w * (nR / self.R0) ** 3)
            w_ = lambda a, b: torch.where(on, a, b)  # noqa: E731
            tm = w_(tm + hp, tm)
            rem = w_(rem - step, rem)
            Rt, Rn, Rp, d1, PG, h = w_(nt, Rt), w_(R, Rn), w_(nR, Rp), w_(nd, d1), w_(nPG, PG), w_(hp, h)
        self.Rt, self.Rp, self.Rn, self.d1, self.PG, self.dtb, self.re = Rt, Rp, Rn, d1, PG, h, rem
        self.PLp = PLp
        return Rt

    # Results -----------------------------------------------------------------
    def output(self, name):
        if name == "p0":
            return self.p0(self.p, self.time)
        if name in ("vx", "vy"):
            return None  # their boundary cells are the package's own layout
        return {"f_g": lambda: self.fg[0], "R_t": lambda: self.Rt, "PG_p": lambda: self.PG,
                "x": lambda: self.pos[-1]}.get(name, lambda: None)()


def _adjoint(case, m):
    m.amp.requires_grad_(True)
    m.phase.requires_grad_(True)
    r, c = focal_radius(case), m.c
    ctr = [focus(c), 0.0] if m.dim == 2 else [0.5 * n * h for n, h in zip(m.n, m.h)]
    d2 = 0.0
    for d in range(m.dim):
        s = [1] * m.dim
        s[d] = -1
        d2 = d2 + ((m.t(np.arange(1.0, m.n[d] + 1)) - 0.5) * m.h[d] - ctr[d]).reshape(s) ** 2
    w = (d2 <= r * r).double() * math.prod(m.h)
    if m.dim == 2:
        w[c.ext_source_row - 1] = 0
        if m.cyl:
            w = w * 2 * math.pi * (m.t(np.arange(1.0, m.n[1] + 1)) - 0.5) * m.h[1]
    J = 0.0
    for _ in range(case["steps"]):
        m.step()
        J = J + m.dt * (w * m.inner(m.p0(m.p, m.time), -1) ** 2).sum()
    J.backward()
    return {"J": float(J), "grad_amp": m.amp.grad, "grad_phase": m.phase.grad}


def exact(case, seed):
    """The 64-bit results; None where the plain form takes too long (driven
    clouds, the 384^3 grid, sweeps, large reverse sweeps) or does not exist
    (rk45, the temperature)."""
    if case["kind"] == "sweep" or case.get("scheme") == "rk45" or case.get("start", 0) > 200:
        return None
    cells = case["x"] * case["y"] * case.get("z", 1)
    if cells > 2e7 or (case["kind"].startswith("adjoint") and cells * case["steps"] > 4.2e8):
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    m = _Model(case, *inputs(case, seed), dev)
    if case["kind"] in ("adjoint2", "adjoint3"):
        return _adjoint(case, m)
    with torch.no_grad():
        for _ in range(case["start"] + case["steps"]):
            m.step()
        fields, bubbles = outputs_of(case)
        return {k: m.output(k) for k in fields + bubbles}
