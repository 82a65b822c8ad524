"""Timed cases of the library: what a simulation program has it do.

The main loop of such a program advances a box by an output interval and then
writes out what the interval produced: the particles and, where the run is
saved, the fluid (reduced vorticity, mean velocity, ion concentrations).  One
pass of a box case is one such interval through the calls that program makes:
`Simulation.step_particles(n)`, then the C ABI readouts into host arrays that
the program keeps.  The other passes are one ensemble interval and one
gradient of the near-contact network.

Families, by the constitutive equations and objects a user can choose:

  ns        Navier_Stokes suspension, with and without thermal kicks or gravity
  el        Electrolyte: charged spheres in a salt, with an external field
  le        Lees-Edwards sheared suspension
  ensemble  independent Navier_Stokes boxes of mixed shapes stepped together
  net       gradient of the near-contact network on a batch of pairs

Both precisions are used: "fp64" throughout, or "mixed" (32-bit fields, 64-bit
particles).  A mixed run's outputs are handed on as 32-bit values, which is
what its fields carry; an fp64 run's as 64-bit ones.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import kapsel_old_b200 as kapsel
from kapsel_old_b200 import nearcontact

_PRECISION = {"fp64": kapsel.FP64, "mixed": kapsel.MIXED}
_KT_SNAP_V, _KT_SNAP_O = 1.439, 1.22


# ---------------------------------------------------------------------------
# the cases
def _box(family, precision, nx, ny, nz, spheres, steps, fluid=True, a=5.0, kbt=1e-3, gravity=0.0):
    return {"family": family, "precision": precision, "nx": nx, "ny": ny, "nz": nz, "spheres": spheres, "a": a,
            "kbt": kbt, "gravity": gravity, "steps": steps, "fluid": fluid}


def listed() -> list:
    return [
        # a host program that calls the step function once per time step and
        # looks at the particles after each (the reference's own main loop
        # with its step replaced): the smallest call, all latency
        dict(_box("ns", "mixed", 64, 64, 64, 16, 1, fluid=False), name="ns_64_each_step"),
        # a small exploratory box, the smallest shape of an ensemble
        dict(_box("ns", "mixed", 32, 32, 32, 8, 200, a=4.0), name="ns_32_mixed"),
        # the plain double-precision suspension: 64^3, 16 spheres, a body force
        dict(_box("ns", "fp64", 64, 64, 64, 16, 200, kbt=0.0, gravity=1e-3), name="ns_64_fp64"),
        # a channel-like box whose axes differ
        dict(_box("ns", "mixed", 64, 64, 128, 40, 200, a=4.5), name="ns_64x64x128_mixed"),
        # the benchmark suspension, 128^3 with 256 spheres, in both precisions
        dict(_box("ns", "mixed", 128, 128, 128, 256, 400), name="ns_128_mixed"),
        dict(_box("ns", "fp64", 128, 128, 128, 256, 200), name="ns_128_fp64"),
        # a large dense suspension (solid fraction 0.27), where the particle
        # kernels and the neighbour lists weigh most
        dict(_box("ns", "mixed", 256, 256, 256, 8600, 150), name="ns_256_dense"),
        # charged spheres: 128^3 with 64 spheres, and a double-precision 64^3
        dict(_box("el", "mixed", 128, 128, 128, 64, 100, kbt=1.0), name="el_128_mixed"),
        dict(_box("el", "fp64", 64, 64, 64, 8, 100, kbt=1.0), name="el_64_fp64"),
        # the benchmark suspension under shear (rheology)
        dict(_box("le", "mixed", 128, 128, 128, 256, 150), name="le_128_mixed"),
        # an ensemble of uneven boxes, as statistics over many small systems need
        {"family": "ensemble", "precision": "mixed", "boxes": 16, "steps": 50, "name": "ensemble_16"},
        # one training step of the near-contact network: forward and backward
        {"family": "net", "precision": "mixed", "rows": 16384, "name": "net_gradient"},
    ]


def draw(rng) -> dict:
    family = rng.choices(["ns", "el", "le", "ensemble", "net"], [5, 2, 2, 1, 1])[0]
    if family == "net":
        return {"family": "net", "precision": "mixed", "rows": int(round(2.0 ** rng.uniform(5.0, 15.0)))}
    if family == "ensemble":
        return {"family": "ensemble", "precision": "mixed", "boxes": rng.randint(3, 16), "steps": rng.randint(10, 50)}
    precision = rng.choice(["fp64", "mixed"])
    # cubes and boxes with uneven axes, up to 128^3 (twice that along an axis
    # of a Navier_Stokes box); every axis holds a few sphere diameters
    lo = 5 if family == "ns" else 6
    p = [rng.randint(lo, 7) for _ in range(3)]
    if rng.random() < 0.4:
        p = [max(p)] * 3
    elif family == "ns" and rng.random() < 0.3:
        p[rng.randrange(3)] = 8
    nx, ny, nz = (1 << q for q in p)
    a = round(rng.uniform(4.0, 5.0 if min(p) == 5 else 6.0), 3)
    # solid fraction over its range, spread over the logarithm
    fraction = 10.0 ** rng.uniform(-2.3, -0.8 if family != "el" else -1.3)
    spheres = max(1, int(fraction * nx * ny * nz / (4.0 / 3.0 * math.pi * a ** 3)))
    most = _sites((nx, ny, nz), a, 1.0)[0].prod()
    spheres = int(min(spheres, 0.8 * most))
    # intervals of some 1e7 to 2e8 grid points in all, 400 steps at most
    steps = int(min(400, max(10, 10.0 ** rng.uniform(7.0, 8.3) / (nx * ny * nz))))
    fluid = rng.random() < 0.85
    if not fluid:
        steps = rng.randint(1, 10)
    # what moves the spheres: the field (el), the shear (le), kicks, or gravity
    # alone, where double precision is what resolves the slow drift
    kbt = 1.0 if family == "el" else rng.choice([1e-3, 1e-2] if precision == "mixed" else [0.0, 1e-3, 1e-2])
    gravity = 1e-3 if family == "ns" and (kbt == 0.0 or rng.random() < 0.3) else 0.0
    return _box(family, precision, nx, ny, nz, spheres, steps, fluid=fluid, a=a, kbt=kbt, gravity=gravity)


# ---------------------------------------------------------------------------
# inputs
def _sites(box, a, gap):
    """Cells per axis of the placement lattice and their widths."""
    n = np.maximum(1, np.floor(np.asarray(box) / (2 * a + gap)).astype(int))
    return n, np.asarray(box) / n


def _place(case, rng) -> np.ndarray:
    """Non-overlapping centres: distinct random sites of a lattice, each moved
    within its cell as far as the minimum surface gap allows (a dense box: 0.05 a,
    else one grid spacing)."""
    box = (case["nx"], case["ny"], case["nz"])
    gap = 1.0 if case["spheres"] <= _sites(box, case["a"], 1.0)[0].prod() else 0.05 * case["a"]
    n, width = _sites(box, case["a"], gap)
    site = rng.permutation(int(n.prod()))[: case["spheres"]]
    ijk = np.stack(np.unravel_index(site, n), axis=1)
    room = np.maximum(0.0, width - (2 * case["a"] + gap))
    x = (ijk + 0.5) * width + (rng.random((len(site), 3)) - 0.5) * room
    return np.mod(x + rng.random(3) * box, box)


_SALT = dict(dielectric=1.0 / (4.0 * math.pi * 0.7), surface_charge=-100.0, debye=4.0, val_p=1.0, val_n=-1.0,
             onsager_p=1.0, onsager_n=1.0, efield=(0.05, 0.0, 0.0))
_SHEAR_RATE = 0.01


def _config(case, seed) -> dict:
    rng = np.random.Generator(np.random.PCG64(seed))
    eq = {"ns": "Navier_Stokes", "el": "Electrolyte", "le": "Shear_Navier_Stokes_Lees_Edwards"}[case["family"]]
    cfg = {"eq": eq, "np_xyz": tuple(int(n).bit_length() - 1 for n in (case["nx"], case["ny"], case["nz"])),
           "a": case["a"], "a_xi": 2.0, "kbt": case["kbt"], "dt": 0.01, "mt_seed": int(seed) & 0x7FFFFFFF,
           "particles": [{"x": tuple(map(float, x))} for x in _place(case, rng)]}
    if case["gravity"]:
        # a body force on the spheres: gravity on a mass excess of 1e-3
        cfg["mass_ratio"] = 1.0 + 1e-3
        cfg["gravity_g"] = case["gravity"] / (4.0 / 3.0 * math.pi * case["a"] ** 3 * 1e-3)
    if case["family"] == "el":
        cfg["alpha_v"] = cfg["alpha_o"] = 0.0
        cfg["electrolyte"] = _SALT
    if case["family"] == "le":
        cfg["shear_rate"] = _SHEAR_RATE
        cfg["start_strain"] = float(0.9 * rng.random())  # somewhere within a shear period
    return cfg


def _ensemble_boxes(case, seed) -> list:
    """Boxes from 32^3, 64^3, 64x64x128 and 128^3 with 1 to 64 spheres of
    radius 4 to 6, the shapes in equal shares; the boxes themselves go with
    the number of boxes, their placements and kicks with the seed."""
    shapes = [(32, 32, 32), (64, 64, 64), (64, 64, 128), (128, 128, 128)]
    rng = np.random.Generator(np.random.PCG64(4))
    seeds = np.random.Generator(np.random.PCG64(seed))
    out = []
    for b in range(case["boxes"]):
        nx, ny, nz = shapes[b % 4]
        a = float(rng.uniform(4.0, 6.0))
        cap = max(1, int(0.1 * nx * ny * nz / (4.0 / 3.0 * math.pi * a ** 3)))
        spheres = min(int(rng.integers(1, 65)), cap, int(_sites((nx, ny, nz), a, 1.0)[0].prod()))
        out.append((_box("ns", "mixed", nx, ny, nz, spheres, case["steps"], a=a), int(seeds.integers(1 << 30))))
    return out


def _net_inputs(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    x = np.zeros((case["rows"], 16), np.float32)
    x[:, :10] = rng.normal(size=(case["rows"], 10))  # standardised features
    y = np.zeros((case["rows"], 16), np.float32)
    y[:, :12] = rng.normal(size=(case["rows"], 12))  # corrections over their RMS
    colw = np.zeros(16, np.float32)
    colw[:12] = 1.0
    return nearcontact.init_params(seed), x, y, colw


class _Run:
    """A box and the host arrays its program reads it into."""

    def __init__(self, case, seed, fluid):
        self.case = case
        cfg = _config(case, seed)
        self.sim = kapsel.Simulation(cfg, _PRECISION[case["precision"]])
        if case["family"] == "le":
            self.sim.set_oblique(cfg["start_strain"], _SHEAR_RATE)
        shape = (2, case["nx"], case["ny"], case["nz"] + 2)
        self.zeta = np.zeros(shape) if fluid else None
        self.conc = np.zeros(shape) if fluid and case["family"] == "el" else None
        self.uk_dc = np.zeros(3)


def prepare(case, seed):
    if case["family"] == "net":
        params, x, y, colw = _net_inputs(case, seed)
        return {"case": case, "net": nearcontact.NearContactNet(params), "x": x, "y": y, "colw": colw}
    if case["family"] == "ensemble":
        boxes = [_Run(c, s, False) for c, s in _ensemble_boxes(case, seed)]
        # the program advances the boxes once before it groups them
        for b in boxes:
            b.sim.step(1)
        return {"case": case, "boxes": boxes, "batch": kapsel.Batch([b.sim for b in boxes])}
    return {"case": case, "run": _Run(case, seed, case["fluid"])}


# ---------------------------------------------------------------------------
# one pass
def _host(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def _kept(case) -> tuple:
    """The particle records a program keeps.  Uniformly charged spheres hardly
    turn, which 32-bit fields resolve to a few digits only."""
    return ("x", "v", "q") if case["family"] == "el" and case["precision"] == "mixed" else ("x", "v", "omega", "q")


def _particles(case, records) -> dict:
    return {k: records[k] for k in _kept(case)}


def run(state):
    case = state["case"]
    if case["family"] == "net":
        grad, loss = state["net"].gradient(state["x"], state["y"], state["colw"])
        return {"grad": grad, "loss": np.float32(loss)}
    as_kept = (lambda a: a.astype(np.float32)) if case["precision"] == "mixed" else (lambda a: a)
    if case["family"] == "ensemble":
        state["batch"].step(case["steps"])
        out = [_particles(case, b.sim.particles()) for b in state["boxes"]]
        return {"msd": as_kept(state["batch"].msd()),
                **{k: as_kept(np.concatenate([p[k] for p in out])) for k in ("x", "v", "omega", "q")}}
    r = state["run"]
    out = _particles(case, r.sim.step_particles(case["steps"]))
    if r.zeta is not None:
        r.sim._check(r.sim.L.kapsel_gpu_get_zeta(r.sim.h, _host(r.zeta), _host(r.uk_dc)))
        out["zeta"] = r.zeta  # the mean velocity is no output: minus the spheres' momentum, which v has
    if r.conc is not None:
        r.sim._check(r.sim.L.kapsel_gpu_get_concentration(r.sim.h, _host(r.conc)))
        out["conc"] = r.conc
    return {k: as_kept(v) for k, v in out.items()}


# ---------------------------------------------------------------------------
# what a pass cannot do without
def _box_work(case) -> dict:
    n = case["nx"] * case["ny"] * case["nz"]
    real = 4 if case["precision"] == "mixed" else 8
    spectrum = math.prod(2 * ((m + 2) // 3) - 1 for m in (case["nx"], case["ny"])) * ((case["nz"] + 2) // 3) * 2 * real
    spectra = 4 if case["family"] == "el" else 2  # reduced vorticity, two concentrations
    transforms = {"ns": 14, "el": 33, "le": 15}[case["family"]]  # real 3D transforms of a step
    record = 35 * 8 * case["spheres"]
    out = (2 * n * 8 * spectra // 2 if case["fluid"] else 0) + record
    stencil = 4.0 / 3.0 * math.pi * (case["a"] + 1.0) ** 3 * case["spheres"]
    return {"bytes": case["steps"] * 2.0 * (spectra * spectrum + record) + out,
            "flops": case["steps"] * (transforms * 2.5 * n * math.log2(n) + 100.0 * stencil)}


def work(case) -> dict:
    if case["family"] == "net":
        weights = 16 * 128 + 2 * 128 * 128 + 128 * 16
        return {"bytes": 4.0 * (32 * case["rows"] + 2 * 37264), "flops": 6.0 * weights * case["rows"]}
    if case["family"] == "ensemble":
        parts = [_box_work(dict(c, fluid=False)) for c, _ in _ensemble_boxes(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    return _box_work(case)


# ---------------------------------------------------------------------------
# the same outputs in 64 bits, by plain torch
_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(a, dtype=torch.float64, device=_DEV)


class _Noise:
    """Normals of the thermostat: MT19937 words mapped to (w + 1/2) / 2^32, two
    at a time through the polar method."""

    def __init__(self, seed):
        self.words = np.random.RandomState(seed)
        self.left = np.zeros((0, 2))

    def pairs(self, n):
        while len(self.left) < n:
            w = self.words.randint(0, 1 << 32, size=(2 * n, 2), dtype=np.uint32).astype(np.float64)
            u = 2.0 * (w + 0.5) / 4294967296.0 - 1.0
            r2 = (u ** 2).sum(1)
            u, r2 = u[(r2 < 1.0) & (r2 > 0.0)], r2[(r2 < 1.0) & (r2 > 0.0)]
            self.left = np.concatenate([self.left, u * np.sqrt(-2.0 * np.log(r2) / r2)[:, None]])
        out, self.left = self.left[:n], self.left[n:]
        return out


class _Exact:
    """A box in 64 bits: the velocity spectrum (rather than the reduced
    vorticity) and the particles, advanced by the smoothed-profile step."""

    def __init__(self, case, seed):
        self.c, self.cfg = case, _config(case, seed)
        self.N = (case["nx"], case["ny"], case["nz"])
        self.L = _t(self.N)
        k = [torch.arange(n, dtype=torch.float64, device=_DEV) for n in (*self.N[:2], self.N[2] // 2 + 1)]
        k[:2] = [torch.where(q > len(q) // 2, q - len(q), q) for q in k[:2]]  # the Nyquist wavenumber is positive
        self.ki = [k[0][:, None, None], k[1][None, :, None], k[2][None, None, :]]
        self.kept = torch.ones((), dtype=torch.bool, device=_DEV)
        for d in range(3):
            self.kept = self.kept & (self.ki[d].abs() < (self.N[d] + 2) // 3)
        self.k = [self.ki[d] * (2.0 * math.pi / self.N[d]) for d in range(3)]
        self.k2 = sum(q * q for q in self.k)
        self.ik2 = torch.where(self.k2 > 0, 1.0 / self.k2, torch.zeros_like(self.k2))
        self.a, self.dt = case["a"], 0.01
        x = _t([p["x"] for p in self.cfg["particles"]])
        z = torch.zeros_like(x)
        self.x, self.v, self.vo, self.w, self.wo, self.fr = x, z, z, z, z, z
        self.q = torch.zeros(len(x), 4, dtype=torch.float64, device=_DEV)
        self.q[:, 0] = 1.0
        self.qo = self.q
        self.mass = self.cfg.get("mass_ratio", 1.0) * 4.0 / 3.0 * math.pi * self.a ** 3
        self.moi = 0.4 * self.mass * self.a ** 2
        m = int(self.a) + 4
        r = torch.arange(-m, m + 1, device=_DEV)
        g = torch.stack(torch.meshgrid(r, r, r, indexing="ij"), -1).reshape(-1, 3)
        self.cells = g[(g.double() ** 2).sum(1).sqrt() < self.a + 1.0 + 1.7321]
        self.noise = _Noise(self.cfg["mt_seed"])
        self.u = torch.zeros((3, *self.kept.shape), dtype=torch.complex128, device=_DEV)
        self.zeta = None
        self.ts, self.deg, self.rate = 0, 0.0, 0.0
        # spheres per chunk of the point-wise work
        self.chunk = 1024

    # forward transforms carry exp(+i k.x), so a derivative is -i k
    def fwd(self, a):
        return torch.fft.rfftn(a, dim=(-3, -2, -1)).conj()

    def inv(self, A):
        return torch.fft.irfftn(A.conj(), s=self.N, dim=(-3, -2, -1))

    def curl(self, A):
        k = self.k
        return torch.stack([-1j * (k[1] * A[2] - k[2] * A[1]), -1j * (k[2] * A[0] - k[0] * A[2]),
                            -1j * (k[0] * A[1] - k[1] * A[0])])

    def solenoidal(self, A):
        d = sum(self.k[i] * A[i] for i in range(3)) * self.ik2
        return torch.stack([A[i] - d * self.k[i] for i in range(3)])

    # --- spheres
    def points(self, x):
        """Grid points around centres x: index, vector from the centre, profile
        and the number of y images crossed."""
        n, sheared = torch.tensor(self.N, device=_DEV), self.c["family"] == "le"
        cell = x.long()
        at = cell[:, None] + self.cells
        r = self.cells.double() - (x - cell)[:, None]
        image = torch.div(at[..., 1], n[1], rounding_mode="floor")
        if sheared:  # the x grid of an image is shifted with it
            xo = torch.remainder(at[..., 0].double() - image * self.deg * self.N[1] + (x - cell)[:, None, 0], self.N[0])
            ix = xo.long().clamp(max=self.N[0] - 1)
            r = r.clone()
            r[..., 0] = self.cells[:, 0].double() - (xo - ix)
            at = torch.stack([ix, at[..., 1], at[..., 2]], -1)
        at = torch.remainder(at, n)
        s = (r ** 2).sum(-1).sqrt()
        inner = self._edge(self.a + 1.0 - s)
        return ((at[..., 0] * n[1] + at[..., 1]) * n[2] + at[..., 2]), r, inner / (inner + self._edge(s - self.a + 1.0)), image

    @staticmethod
    def _edge(y):
        return torch.where(y > 0, torch.exp(-1.0 / torch.where(y > 0, y, torch.ones_like(y)) ** 2), torch.zeros_like(y))

    def rigid(self, s, r, image):
        v = self.v[s][:, None] + torch.linalg.cross(self.w[s][:, None].expand_as(r), r)
        if self.c["family"] == "le":
            v = v.clone()
            v[..., 0] -= image * self.rate * self.N[1]
        return v

    def spheres(self):
        for i in range(0, len(self.x), self.chunk):
            yield slice(i, min(i + self.chunk, len(self.x)))

    def profile(self, value, n):
        """Sum over the spheres of n fields of point values."""
        out = torch.zeros(n, math.prod(self.N), dtype=torch.float64, device=_DEV)
        for s in self.spheres():
            at, r, ph, image = self.points(self.x[s])
            for d, val in enumerate(value(s, r, ph, image)):
                out[d].index_add_(0, at.reshape(-1), val.reshape(-1))
        return out.reshape(n, *self.N)

    def rigidity(self, u):
        f = self.profile(lambda s, r, ph, im: [ph, *(self.rigid(s, r, im) * ph[..., None]).unbind(-1)], 4)
        phi, up = f[0], f[1:]
        over = phi.clamp(min=1.0)
        return up / over - phi / over * u

    def hydro(self, u):
        u = u.reshape(3, -1)
        force, torque = [], []
        for s in self.spheres():
            at, r, ph, image = self.points(self.x[s])
            f = (self.rigid(s, r, image) - u[:, at].permute(1, 2, 0)) * ph[..., None]
            force.append(f.sum(1))
            torque.append(torch.linalg.cross(r, f).sum(1))
        return -torch.cat(force) / self.dt, -torch.cat(torque) / self.dt

    def pair_forces(self):
        out = torch.zeros_like(self.x)
        dia = 2.0 * self.a
        if self.c["family"] == "le":
            dia = min((dia + 2.0) / 2.0 ** (1.0 / 6.0), dia)
        cells = torch.div(self.x, 16.0, rounding_mode="floor")
        nc = self.L.new_tensor([n // 16 for n in self.N])
        for s in self.spheres():
            d = self.x[None] - self.x[s][:, None]
            y = d[..., 1] - torch.round(d[..., 1] / self.L[1]) * self.L[1]
            if self.c["family"] == "le":
                d = d.clone()
                d[..., 0] -= torch.round((d[..., 1] - y) / self.L[1]) * self.deg * self.L[1]
            d = d - torch.round(d / self.L) * self.L
            r2 = (d ** 2).sum(-1)
            i, j = torch.nonzero((r2 > 0) & (r2 < (dia * 2.0 ** (1.0 / 6.0)) ** 2), as_tuple=True)
            r2, d = r2[i, j], d[i, j]
            p6 = (dia * dia / r2) ** 3
            f = 24.0 / r2 * (2.0 * p6 * p6 - p6)
            if self.c["family"] != "le":
                # a pair is met once for each neighbouring 16-wide cell that is the partner's
                hi = torch.maximum(i + s.start, j)
                lo = torch.minimum(i + s.start, j)
                for axis in range(3):
                    met = 0.0
                    for o in (-1.0, 0.0, 1.0):
                        met = met + (torch.remainder(cells[hi, axis] + o, nc[axis]) == cells[lo, axis]).double()
                    f = f * met
            out.index_add_(0, i + s.start, -f[:, None] * d)
        if self.c["gravity"]:
            out[:, 2] -= self.c["gravity"]
        return out

    def move(self):
        first, h = self.ts == 0, 0.5 * self.dt
        x = self.x + (self.dt * self.v if first else h * (3.0 * self.v - self.vo))
        if self.c["family"] == "le":
            image = torch.div(x[:, 1], self.L[1], rounding_mode="floor")
            x[:, 0] -= image * self.deg * self.L[1]
            jump = torch.zeros_like(x)
            jump[:, 0] = -image * self.rate * self.L[1]
            self.v, self.vo = self.v + jump, self.vo + jump
        self.x = torch.remainder(x, self.L)
        if first:
            dq, qo = _qmul(_qvec(self.w), self.q) * 0.5 * self.dt, self.q
        else:
            turn = 3.0 * _to_body(self.w, self.q) - _to_body(self.wo, self.qo)
            dq, qo = _qmul(self.q, _qvec(turn)) * 0.5 * h, self.q
        q = self.q + dq
        self.q, self.qo = q / q.norm(dim=1, keepdim=True), qo

    def kick(self, f, t):
        fr = self.pair_forces()
        vo, wo = self.v, self.w
        pair = fr if self.ts == 0 else 0.5 * (fr + self.fr)
        self.v = self.v + self.dt / self.mass * (f + pair)
        self.w = self.w + self.dt / self.moi * t
        self.vo, self.wo, self.fr = vo, wo, fr
        kbt = self.c["kbt"]
        if kbt > 0.0 and self.c["family"] != "el":
            g = _t(self.noise.pairs(3 * len(self.x)).reshape(-1, 6))
            drag = 6.0 * math.pi * self.a
            self.v = self.v + g[:, :3] * (_KT_SNAP_V * math.sqrt(drag * self.dt * kbt) / self.mass)
            drag = 8.0 * math.pi * self.a ** 3
            self.w = self.w + g[:, 3:] * (_KT_SNAP_O * math.sqrt(drag * self.dt * kbt) / self.moi)

    # --- fluid
    def momentum(self, u):
        """Solenoidal part of -(u.grad)u, retained modes."""
        out = [0.0, 0.0, 0.0]
        for i in range(3):
            for j in range(i, 3):
                p = self.fwd(u[i] * u[j])
                out[i] = out[i] + 1j * self.k[j] * p
                if i != j:
                    out[j] = out[j] + 1j * self.k[i] * p
        return self.solenoidal(torch.stack(out)) * self.kept

    def step_ns(self):
        mean = self.u[:, 0, 0, 0].clone()
        adv = self.momentum(self.inv(self.u))
        self.u = self.u + torch.expm1(-self.k2 * self.dt) * (self.u - adv * self.ik2)
        self.u[:, 0, 0, 0] = mean
        self.finish(self.inv(self.u))

    def finish(self, u):
        self.move()
        self.kick(*self.hydro(u))
        self.add(self.rigidity(u))

    def add(self, f):
        f = self.solenoidal(self.fwd(f) * self.kept)
        f[:, 0, 0, 0] = f[:, 0, 0, 0].real.to(f.dtype)
        self.u = self.u + f

    # --- ions
    def start_el(self):
        phi = self.profile(lambda s, r, ph, im: [ph], 1)[0]
        free = float((1.0 - phi).sum())
        z, n = _SALT["surface_charge"], len(self.x)
        bulk = self.c["kbt"] * _SALT["dielectric"] / _SALT["debye"] ** 2 / 2.0
        c = [(-z * n if z < 0 else 0.0) / free + bulk, (z * n if z > 0 else 0.0) / free + bulk]
        self.total = [q * free for q in c]
        self.conc = torch.stack([self.fwd(torch.full(self.N, q, dtype=torch.float64, device=_DEV)) for q in c])

    def charges(self, normal):
        def values(s, r, ph, im):
            d = (r ** 2).sum(-1).sqrt()
            near = ((d - self.a).abs() < 1.0).double()
            out = [ph, _SALT["surface_charge"] * near * math.pi / 4.0 * torch.cos(math.pi * (self.a - d) / 2.0)]
            return out + [r[..., i] / d.clamp(min=1e-300) * near for i in range(3)] if normal else out

        f = self.profile(values, 5 if normal else 2)
        f[1] *= abs(_SALT["surface_charge"]) * len(self.x) / float(f[1].abs().sum())
        return f

    def charge(self, f, c):
        return f[1] + (c[0] - c[1]) * (1.0 - f[0])

    def step_el(self):
        e = _SALT["efield"]
        f = self.charges(True)
        c = self.inv(self.conc)
        psi = self.fwd(self.charge(f, c)) * self.ik2 / _SALT["dielectric"] * self.kept
        grad = torch.stack([self.inv(-1j * self.k[d] * psi) - e[d] for d in range(3)])
        u = self.inv(self.u)
        normal, n2 = f[2:], (f[2:] ** 2).sum(0)
        n2 = torch.where(n2 > 0, n2, torch.ones_like(n2))
        new = []
        for s, ve in enumerate((1.0, -1.0)):
            flux = torch.stack([self.inv(-1j * self.k[d] * self.c["kbt"] * self.conc[s]) for d in range(3)])
            flux = flux + c[s] * ve * grad
            flux = flux - normal * ((flux * normal).sum(0) / n2) - c[s] * u
            div = sum(-1j * self.k[d] * self.fwd(flux[d]) for d in range(3)) * self.kept
            new.append(self.conc[s] + self.dt * div)
        self.conc = torch.stack(new)
        mean = self.u[:, 0, 0, 0].clone()
        self.u = self.u + self.dt * (self.momentum(u) - self.k2 * self.u)
        self.u[:, 0, 0, 0] = mean
        self.move()
        f = self.charges(False)
        for s in range(2):
            self.conc[s] *= self.total[s] / float(((1.0 - f[0]) * self.inv(self.conc[s])).sum())
        q = self.charge(f, self.inv(self.conc))
        psi = self.fwd(q) * self.ik2 / _SALT["dielectric"]
        force = torch.stack([q * (e[d] - self.inv(self._half(-1j * self.k[d] * psi, d))) for d in range(3)])
        self.add(force * self.dt)
        u = self.inv(self.u)
        self.kick(*self.hydro(u))
        self.add(self.rigidity(u))

    def _half(self, A, d):
        """The full spectrum of a derivative as a half-spectrum inverse reads
        it: of the Nyquist planes along the derivative's axis, which have no
        real inverse, it takes one half and assumes the other its conjugate."""
        nx, ny, _ = self.N
        i = torch.arange(nx, device=_DEV)[:, None]
        j = torch.arange(ny, device=_DEV)[None, :]
        ends = (j == 0) | (j == ny // 2)
        own = ((i == 0) | (i == nx // 2)) & ends
        A = A.clone()
        for plane, keep in ((0, ((j > 0) & (j < ny // 2)) | (ends & (i <= nx // 2))),
                            (self.N[2] // 2, (j > ny // 2) | (ends & (i >= nx // 2)))):
            p = A[:, :, plane]
            partner = p[(-i) % nx, (-j) % ny].conj()
            p = torch.where(keep, p, partner)
            A[:, :, plane] = torch.where(own, p.real.to(p.dtype), p)
        return A

    # --- shear: contravariant components on a grid that deforms with the flow
    def start_le(self):
        self.deg, self.rate = self.cfg["start_strain"], _SHEAR_RATE
        self.zeta = torch.zeros((2, *self.kept.shape), dtype=torch.complex128, device=_DEV)
        self.mean = torch.zeros(3, dtype=torch.float64, device=_DEV)

    def oblique_k2(self):
        k2 = self.k[0] ** 2 + (self.k[1] - self.deg * self.k[0]) ** 2 + self.k[2] ** 2
        return k2, torch.where(k2 > 0, 1.0 / k2, torch.zeros_like(k2))

    def covariant(self, a):
        return torch.stack([a[0] + self.deg * a[1], self.deg * a[0] + (1.0 + self.deg ** 2) * a[1], a[2]])

    def oblique_vorticity(self):
        (kx, ky, kz), (z0, z1) = self.k, self.zeta
        has_x, has_z = self.ki[0] != 0, self.ki[2] != 0
        one = torch.ones_like(self.k2)
        w0 = torch.where(has_x, -(ky * z0 + kz * z1) / torch.where(has_x, kx * one, one), torch.where(has_z, z1, z0))
        w1 = torch.where(has_x | has_z, z0, torch.zeros_like(z0))
        w2 = torch.where(~has_x & has_z, -(ky / torch.where(has_z, kz * one, one)) * z0, z1)
        return torch.stack([w0, w1, w2])

    def oblique_reduce(self, w):
        has_x, has_z = self.ki[0] != 0, self.ki[2] != 0
        z0 = torch.where(has_x | has_z, w[1], w[0])
        z1 = torch.where(~has_x & has_z, w[0], w[2])
        return torch.stack([z0, z1]) * self.kept

    def oblique_velocity(self, w):
        u = self.curl(self.covariant(w)) * self.oblique_k2()[1]
        u[:, 0, 0, 0] = self.mean.to(u.dtype)
        return u

    def rows(self, f, shift):
        """Row y = j of f moved along x by shift[j] cells, linearly between grid points."""
        i = torch.arange(self.N[0], device=_DEV)[:, None]
        j = torch.arange(self.N[1], device=_DEV)[None, :]
        base = torch.floor(shift)
        part = (shift - base)[None, :, None]
        at = torch.remainder(i + base.long()[None], self.N[0])
        return (1.0 - part) * f[:, at, j] + part * f[:, torch.remainder(at + 1, self.N[0]), j]

    def step_le(self):
        k2, ik2 = self.oblique_k2()
        w = self.oblique_vorticity()
        uk = self.oblique_velocity(w)
        adv = self.fwd(torch.linalg.cross(self.inv(uk), self.inv(w), dim=0))
        adv[0] -= 2.0 * self.rate * uk[1]
        adv[1] -= 2.0 * self.rate * self.deg * uk[1]
        f = self.oblique_reduce(self.curl(adv))
        self.zeta = self.zeta + torch.expm1(-k2 * self.dt) * (self.zeta - f * ik2)
        self.mean[1] = 0.0
        u = self.inv(self.oblique_velocity(self.oblique_vorticity()))
        self.deg += _SHEAR_RATE * self.dt
        y = torch.arange(self.N[1], dtype=torch.float64, device=_DEV) - self.N[1] / 2.0
        if self.deg >= 1.0:  # the grid is taken back by one cell per row
            self.deg -= 1.0
            u = self.rows(torch.stack([u[0] + u[1], u[1], u[2]]), -y)
        cart = self.rows(u, -self.deg * y)
        cart[0] += self.deg * cart[1] + _SHEAR_RATE * y[None, :, None]
        self.rate = float((cart[0, :, -1] - cart[0, :, 0]).mean() / (self.N[1] - 1))
        self.move()
        self.kick(*self.hydro(cart))
        f = self.rows(self.rigidity(cart), self.deg * y)
        uk = self.fwd(u + torch.stack([f[0] - self.deg * f[1], f[1], f[2]])) * self.kept
        k2, ik2 = self.oblique_k2()
        k, d = self.k, self.deg
        div = sum(k[i] * uk[i] for i in range(3)) * ik2
        uk = torch.stack([uk[0] - div * ((1.0 + d * d) * k[0] - d * k[1]), uk[1] - div * (k[1] - d * k[0]),
                          uk[2] - div * k[2]])
        self.mean = uk[:, 0, 0, 0].real.clone()
        self.zeta = self.oblique_reduce(self.curl(self.covariant(uk)))
        self.zeta[:, 0, 0, 0] = 0.0

    # --- outputs
    def advance(self, steps):
        if self.c["family"] != "ns":
            getattr(self, "start_" + self.c["family"])()
        for _ in range(steps):
            getattr(self, "step_" + self.c["family"])()
            self.ts += 1

    def packed(self, A):
        """Interleaved rows, zero outside the retained modes."""
        return torch.view_as_real((A * self.kept).resolve_conj()).reshape(*A.shape[:-1], -1).cpu().numpy()

    def outputs(self):
        out = {k: getattr(self, "w" if k == "omega" else k).cpu().numpy() for k in _kept(self.c)}
        if not self.c["fluid"]:
            return out
        if self.zeta is None:
            w = self.curl(self.u)
            has_x, has_y = self.ki[0] != 0, self.ki[1] != 0
            zeta = torch.stack([torch.where(has_x, w[1], torch.where(has_y, w[2], w[0])),
                                torch.where(has_x, w[2], torch.where(has_y, w[0], w[1]))])
        else:
            zeta = self.zeta
        out["zeta"] = self.packed(zeta)
        if self.c["family"] == "el":
            out["conc"] = self.packed(self.conc)
        return out


def _qvec(v):
    return torch.cat([torch.zeros_like(v[:, :1]), v], 1)


def _qmul(a, b):
    s = a[:, :1] * b[:, :1] - (a[:, 1:] * b[:, 1:]).sum(1, keepdim=True)
    return torch.cat([s, a[:, :1] * b[:, 1:] + b[:, :1] * a[:, 1:] + torch.linalg.cross(a[:, 1:], b[:, 1:])], 1)


def _to_body(v, q):
    conj = torch.cat([q[:, :1], -q[:, 1:]], 1)
    return _qmul(_qmul(conj, _qvec(v)), q)[:, 1:]


def _exact_net(case, seed):
    params, x, y, colw = (_t(a) for a in _net_inputs(case, seed))
    params.requires_grad_(True)
    at, h = 0, x
    for i, (o, n) in enumerate(((128, 16), (128, 128), (128, 128), (16, 128))):
        weight, at = params[at: at + o * n].reshape(o, n), at + o * n
        h, at = h @ weight.T + params[at: at + o], at + o
        h = h if i == 3 else torch.nn.functional.silu(h)
    loss = (colw * (h - y) ** 2).sum() / case["rows"]
    loss.backward()
    return {"grad": params.grad.cpu().numpy(), "loss": float(loss)}


def exact(case, seed):
    if case["family"] == "net":
        return _exact_net(case, seed)
    if case["family"] == "ensemble":
        out = []
        for c, s in _ensemble_boxes(case, seed):
            e = _Exact(dict(c, fluid=False), s)
            e.advance(1)
            start, moved = e.x, torch.zeros_like(e.x)
            for _ in range(case["steps"]):
                before = e.x
                e.advance(1)
                step = e.x - before
                moved = moved + step - torch.round(step / e.L) * e.L
            out.append((float((moved ** 2).sum(1).mean()), e.outputs()))
        return {"msd": np.array([m for m, _ in out]),
                **{k: np.concatenate([o[k] for _, o in out]) for k in ("x", "v", "omega", "q")}}
    e = _Exact(case, seed)
    e.advance(case["steps"])
    return e.outputs()
