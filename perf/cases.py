"""Performance cases of the FDTD step path: what a user's program has it do.

Every case steps scenes through the package's public entry points
(``B200FDTD``, ``B200Batch``, ``adjoint.design_monitors``) over the sizes, media,
boundaries, storage types and directions that the workloads and tests of this
repository use.  ``exact`` restates the path with dense 64-bit torch tensors.
"""
import dataclasses
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path.cwd()
NAME = "witwin_maxwell_b200"


def _package():
    if NAME not in sys.modules:
        folder = ROOT / "witwin-maxwell_b200"
        spec = importlib.util.spec_from_file_location(NAME, folder / "__init__.py",
                                                      submodule_search_locations=[str(folder)])
        module = importlib.util.module_from_spec(spec)
        sys.modules[NAME] = module
        spec.loader.exec_module(module)
    return sys.modules[NAME]


wm = _package()
COMPONENTS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
ETA_0 = 376.730313668
DEVICE = "cuda"


# --------------------------------------------------------------------------
# Cases
# --------------------------------------------------------------------------
def listed():
    return [
        # a first look at a scene: the smallest grid a user steps, where launches and latency count
        dict(name="tiny_dipole", kind="steps", scene="dipole", nx=24, ny=20, nz=18, pml=5, steps=256, storage="fp32"),
        # one whole solve of a small scene: engine build, stepping, spectra on the host
        dict(name="solve_64", kind="solve", scene="dipole", nx=64, ny=64, nz=64, pml=10, steps=400, storage="fp32"),
        # a closed cavity with ragged sides: no absorber, one probe
        dict(name="cavity_odd", kind="steps", scene="cavity", nx=181, ny=211, nz=157, pml=0, steps=128, storage="fp32"),
        # the common case: dielectric parts in an absorbing box, a plane monitor
        dict(name="cpml_192", kind="steps", scene="dielectric", nx=192, ny=192, nz=160, pml=10, steps=128,
             storage="fp32"),
        # the same on a graded grid (spacing varies along every axis), ragged sides
        dict(name="graded_odd", kind="steps", scene="graded", nx=139, ny=117, nz=171, pml=8, steps=128, storage="fp32"),
        # dispersive sphere and slab in a TFSF plane wave, 16-frequency flux box: odd and full size
        dict(name="dispersive_131", kind="steps", scene="dispersive", nx=131, ny=131, nz=131, pml=12, steps=128,
             storage="fp32"),
        dict(name="dispersive_256", kind="steps", scene="dispersive", nx=256, ny=256, nz=256, pml=12, steps=64,
             storage="fp32"),
        # a Bloch-periodic grating (complex field) driven by its TFSF slab
        dict(name="grating_256", kind="steps", scene="grating", nx=256, ny=256, nz=192, pml=16, steps=48, storage="fp32"),
        # fields stored in 16 bits
        dict(name="bf16_160", kind="steps", scene="dispersive", nx=160, ny=160, nz=160, pml=12, steps=48,
             storage="bf16"),
        # a sweep of independent designs stepped together
        dict(name="batch_8", kind="batch", scene="designs", nx=128, ny=128, nz=128, pml=8, steps=128, scenes=8,
             storage="fp32"),
        # one iteration of inverse design (forward and adjoint gradient): stored history, checkpoint replay
        dict(name="design_80", kind="design", scene="design", nx=80, ny=80, nz=48, pml=10, steps=400, stride=0,
             storage="fp32"),
        dict(name="design_160", kind="design", scene="design", nx=160, ny=160, nz=96, pml=10, steps=800, stride=50,
             storage="fp32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ranges: 18 to 256 cells a side, every scene kind, option and direction."""
    what = rng.choice(["dipole", "dipole", "solve", "cavity", "dielectric", "graded", "dispersive", "dispersive",
                       "grating", "reduced", "batch", "design"])
    if what == "design":
        scale = rng.choice([1, 2])
        return dict(kind="design", scene="design", nx=160 // scale, ny=160 // scale, nz=96 // scale, pml=10,
                    steps=rng.randrange(200, 800 if scale == 1 else 400), stride=rng.choice([0, rng.randrange(25, 101)]),
                    storage="fp32")
    if what == "batch":
        top = rng.randrange(72, 129)
        return dict(kind="batch", scene="designs", nx=top, ny=top, nz=top, pml=8, steps=rng.randrange(64, 129),
                    scenes=rng.randrange(2, 9), storage="fp32")
    if what in ("dispersive", "reduced"):
        n = rng.randrange(96, 257 if what == "dispersive" else 193)
        return dict(kind="steps", scene="dispersive", nx=n, ny=n, nz=n, pml=12, steps=rng.randrange(24, 65 if what == "dispersive" else 49),
                    storage="fp32" if what == "dispersive" else rng.choice(["bf16", "fp16"]))
    if what == "grating":
        return dict(kind="steps", scene="grating", nx=16 * rng.randrange(4, 17), ny=_log(rng, 48, 256),
                    nz=_log(rng, 112, 192), pml=16, steps=rng.randrange(24, 49), storage=rng.choice(["fp32", "fp32", "bf16"]))
    lo, hi = {"dipole": (18, 64), "solve": (32, 96), "cavity": (24, 256), "dielectric": (64, 224),
              "graded": (64, 192)}[what]
    sides = [_log(rng, lo, hi) for _ in range(3)]
    pml = {"dipole": 5, "solve": 10, "cavity": 0, "dielectric": rng.choice([8, 10, 12]), "graded": 8}[what]
    return dict(kind="solve" if what == "solve" else "steps", scene="dipole" if what == "solve" else what,
                nx=sides[0], ny=sides[1], nz=sides[2], pml=pml,
                steps=rng.randrange(200, 401) if what == "solve" else rng.randrange(64, 129), storage="fp32")


# --------------------------------------------------------------------------
# Scenes
# --------------------------------------------------------------------------
PASSES = 16  # passes of a run: step tables cover PASSES * steps steps


def _pulse(rng, dt, steps):
    return wm.GaussianPulse(300e12, 100e12, amplitude=float(rng.uniform(0.5, 2.0)), phase=float(rng.uniform(0, 6)),
                            delay=0.5 * steps * dt)


def _scene(case, rng):
    cells = (case["nx"], case["ny"], case["nz"])
    pml, steps = case["pml"], case["steps"]
    mid = tuple(c // 2 for c in cells)
    W = wm.workloads
    if case["scene"] == "dispersive":
        sc = W.dispersive_256(cells[0], pml, slab_through_pml=False)
        sc.sources = [dataclasses.replace(sc.sources[0], source_time=_pulse(rng, sc.resolve_dt(), steps))]
        return sc
    if case["scene"] == "grating":
        sc = W.bloch_grating(cells, pml)
        pulse = dataclasses.replace(_pulse(rng, sc.resolve_dt(), steps), fwidth=120e12)
        sc.sources = [dataclasses.replace(sc.sources[0], source_time=pulse)]
        return sc
    if case["scene"] == "design":
        return W.adjoint_160(steps, scale=160 // cells[0])
    sc = wm.Scene(cells=cells, spacing=25e-9, pml_cells=pml)
    freqs = (250e12, 300e12, 350e12)
    third = [max(2, (c - 2 * pml) // 3) for c in cells]
    lo = tuple(m - t // 2 for m, t in zip(mid, third))
    hi = tuple(a + t for a, t in zip(lo, third))
    if case["scene"] == "cavity":
        sc.boundary = (wm.BOUNDARY_PEC,) * 6
    else:
        sc.structures.append(wm.Structure(wm.Box(lo, hi), wm.Medium(eps_r=float(rng.uniform(2.0, 6.0)))))
        if case["scene"] == "dipole":
            sc.monitors.append(wm.PlaneMonitor("plane", 2, mid[2] + 1, frequencies=freqs))
        else:
            sc.structures.append(wm.Structure(wm.Sphere(tuple(float(v) for v in hi), min(third) / 3.0),
                                              wm.Medium(eps_r=2.25, eps_diag=(2.25, 2.5, 2.0))))
            sc.monitors.append(wm.flux_monitor("flux", 2, mid[2] + 3, freqs))
    sc.sources.append(wm.PointDipole(mid, "Ez", _pulse(rng, sc.resolve_dt(), steps), width=25e-9))
    sc.monitors.append(wm.PointMonitor("point", tuple(m + 1 for m in mid), frequencies=freqs))
    return sc


def _graded(cs):
    """The compiled scene on a grid whose spacing widens by up to 30 % away from the middle."""
    inv_e, inv_h = [], []
    for n in cs.nodes:
        t = np.linspace(-1.0, 1.0, n)
        node = 1.0 + 0.3 * t * t
        inv_e.append((np.float64(cs.inv_e[0][0]) / node).astype(np.float32))
        inv_h.append((np.float64(cs.inv_h[0][0]) / (0.5 * (node[1:] + node[:-1]))).astype(np.float32))
    return dataclasses.replace(cs, inv_e=inv_e, inv_h=inv_h)


def _compiled(case, seed):
    """The solver scenes of a case (more than one for a batch)."""
    rng = np.random.default_rng([seed, 1])
    if case["kind"] == "batch":
        # the sizes belong to the case, the sources to the seed
        scenes = wm.workloads.batched_designs(case["scenes"], seed=1, size_range=(64, case["nx"]), pml=case["pml"])
        for sc in scenes:
            sc.sources = [dataclasses.replace(sc.sources[0], source_time=_pulse(rng, sc.resolve_dt(), case["steps"]))]
        return [wm.compile_scene(sc, PASSES * case["steps"]) for sc in scenes]
    total = case["steps"] if case["kind"] == "solve" else PASSES * case["steps"]
    cs = wm.compile_scene(_scene(case, rng), total)
    return [_graded(cs) if case["scene"] == "graded" else cs]


def _field(cs, name, seed, dtype=torch.float32):
    """A smooth field that vanishes on the outer faces: a few standing waves, O(1) for E, O(1 / eta0) for H."""
    rng = np.random.default_rng([seed, 2, COMPONENTS.index(name)])
    shape = wm.scene.component_shape(name, cs.nodes)
    out = torch.zeros(shape, dtype=torch.float32, device=DEVICE)
    for _ in range(3):
        amp = rng.uniform(-1, 1) / (1.0 if name[0] == "E" else ETA_0)
        factors = []
        for n in shape:
            t = torch.linspace(0, 1, n, dtype=torch.float64, device=DEVICE)
            w = torch.sin(math.pi * int(rng.integers(2, 2 + max(2, n // 12))) * t)
            w[-1] = 0.0
            factors.append(w.to(torch.float32))
        out += float(amp) * factors[0][:, None, None] * factors[1][None, :, None] * factors[2][None, None, :]
    return out.to(dtype)


def _design_eps(case, seed):
    s = 160 // case["nx"]
    gen = torch.Generator().manual_seed(int(seed))
    eps = 1.0 + 11.0 * torch.rand((64 // s, 64 // s, 16 // s), generator=gen, dtype=torch.float64)
    return eps.to(device=DEVICE, dtype=torch.float32)


DESIGN_KEYS = (("patch", "Ex"), ("patch", "Ey"), ("patch", "Ez"))


# --------------------------------------------------------------------------
# prepare / run
# --------------------------------------------------------------------------
def prepare(case, seed):
    state = {"case": case, "n": 0}
    if case["kind"] == "design":
        sc = _scene(case, np.random.default_rng([seed, 1]))
        history = dict(history="replay", stride=case["stride"]) if case["stride"] else dict(history="store")
        state["problem"] = wm.adjoint.DesignProblem(sc, case["steps"], **history)
        state["eps"] = _design_eps(case, seed)
        return state
    compiled = _compiled(case, seed)
    if case["kind"] == "solve":
        state["compiled"] = compiled[0]
        return state
    solvers = []
    for at, cs in enumerate(compiled):
        solver = wm.B200FDTD(cs, storage=case["storage"], storage_scales=_scales(case)).init_field()
        for name in COMPONENTS:
            solver.set_field(name, _field(cs, name, seed + 1000 * at))
        solvers.append(solver)
    state["solvers"] = solvers
    if case["kind"] == "batch":
        state["batch"] = wm.B200Batch(solvers)
    return state


def _scales(case):
    """FP16 storage: scales for fields of up to 2^5 (E), the others take the engine's own."""
    return [2.0 ** -10] * 3 + [2.0 ** -18] * 3 if case["storage"] == "fp16" else None


def _outputs(solver, whole):
    """The fields and the monitor spectra; a batch's spectra in one tensor for each scene."""
    out = {}
    spectra = solver.monitor_results()
    if whole:
        out["spectra"] = spectra
    else:
        out["spectra"] = torch.cat([v.reshape(-1) for m in spectra.values() for v in m.values()])
    out["fields"] = {name: solver.field(name) for name in COMPONENTS}
    if solver.handle_imag is not None:
        out["imag"] = {name: solver.field(name, imag=True) for name in COMPONENTS}
    return out


def run(state):
    case = state["case"]
    steps = case["steps"]
    if case["kind"] == "design":
        eps = state["eps"].clone().requires_grad_(True)
        spectra = wm.adjoint.design_monitors(eps, state["problem"], DESIGN_KEYS)
        loss = sum(v.abs().square().sum() for v in spectra["patch"].values())
        loss.backward()
        return {"spectra": {k: v.detach() for k, v in spectra["patch"].items()}, "grad": eps.grad}
    if case["kind"] == "solve":
        solver = wm.B200FDTD(state["compiled"], storage=case["storage"]).init_field()
        solver.step_range(0, steps)
        out = {"spectra": solver.monitor_results(host=True),
               "fields": {name: solver.field(name) for name in COMPONENTS}}
        solver.close()
        return out
    n = state["n"]
    state["n"] = (n + steps) % (PASSES * steps)
    if case["kind"] == "batch":
        state["batch"].step_range(n, n + steps)
        return [_outputs(s, False) for s in state["solvers"]]
    solver = state["solvers"][0]
    solver.step_range(n, n + steps)
    return _outputs(solver, True)


# --------------------------------------------------------------------------
# work / tolerance
# --------------------------------------------------------------------------
def _step_cost(cells, case, sides):
    """Bytes and operations of one step of `cells` cells: every state array read and written once."""
    word = 4 if case["storage"] == "fp32" else 2
    scene = case["scene"]
    share = sum(2.0 * case["pml"] / n for n in (sides[2:] if scene == "grating" else sides))
    # fields, CPML state (four arrays an axis over its slabs), E coefficients
    per = 12 * word + 32.0 * share + (0 if scene == "cavity" else 12)
    flops = 36 + 12 * share
    if scene == "dispersive":
        # sphere of radius 60/256 with P and J, slab of 40/256 (inside the absorber) with J; three components each
        sphere = 4.0 / 3.0 * math.pi * (60.0 / 256.0) ** 3
        slab = 40.0 / 256.0 * (1.0 - 2.0 * case["pml"] / sides[1]) * (1.0 - 2.0 * case["pml"] / sides[2])
        per += 3 * 2 * word * (2 * sphere + slab)
        flops += 3 * (8 * sphere + 6 * slab)
    if scene == "grating":
        per += 3 * 2 * word / 24.0  # half of a layer of 32 in 384 cells
    return cells * per, cells * flops


def work(case):
    sides = (case["nx"], case["ny"], case["nz"])
    if case["kind"] == "batch":
        scenes = wm.workloads.batched_designs(case["scenes"], seed=1, size_range=(64, case["nx"]), pml=case["pml"])
        costs = [_step_cost(float(np.prod(s.cells)), case, s.cells) for s in scenes]
    else:
        costs = [_step_cost(float(np.prod(sides)), case, sides)]
    bytes_, flops = (sum(c[k] for c in costs) * case["steps"] for k in (0, 1))
    if case["scene"] == "grating":
        bytes_, flops = 2 * bytes_, 2 * flops  # real and imaginary channel
    if case["kind"] == "design":
        # the forward steps, the reverse steps and, from checkpoints, the replayed ones
        times = 3 if case["stride"] else 2
        bytes_, flops = times * bytes_, times * flops
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """About four times the error against ``exact`` (the largest output's)."""
    if case["storage"] != "fp32":
        # every step rounds the fields to 16 bits; a change of the 32-bit sums moves some of the roundings
        return {"rel": 3e-2 if case["storage"] == "bf16" else 8e-3}
    if case["kind"] == "solve":
        # an Ez dipole leaves little behind after 400 steps: 6e-5 in Hz
        return {"rel": 2.3e-4}
    if case["kind"] == "design":
        # the components across the beam's polarisation are small: 4e-6 in Ex
        return {"rel": 2e-5}
    return {"rel": 5e-6}


# --------------------------------------------------------------------------
# The same path in 64 bits, with dense torch tensors
# --------------------------------------------------------------------------
# component -> ((axis, field, sign) of its two curl terms)
H_CURL = {"Hx": ((1, "Ez", -1), (2, "Ey", 1)), "Hy": ((0, "Ez", 1), (2, "Ex", -1)), "Hz": ((0, "Ey", -1), (1, "Ex", 1))}
E_CURL = {"Ex": ((1, "Hz", 1), (2, "Hy", -1)), "Ey": ((0, "Hz", -1), (2, "Hx", 1)), "Ez": ((0, "Hy", 1), (1, "Hx", -1))}


def _along(values, axis):
    shape = [1, 1, 1]
    shape[axis] = -1
    return values.reshape(shape)


def _box(b):
    return slice(b[0], b[1]), slice(b[2], b[3]), slice(b[4], b[5])


class _Dense:
    """One scene: fields, CPML and pole state as full arrays (complex on Bloch faces)."""

    def __init__(self, cs):
        self.cs = cs
        self.wave = any(b == wm.BOUNDARY_BLOCH for b in cs.boundary)
        self.kind = torch.complex128 if self.wave else torch.float64
        self.F = {n: torch.zeros(wm.scene.component_shape(n, cs.nodes), dtype=self.kind, device=DEVICE)
                  for n in COMPONENTS}
        self.psi = {}
        self.decay, self.curl = {}, {}
        for n in COMPONENTS:
            d, c = cs.uniform[n]
            self.decay[n] = d if cs.decay[n] is None else self.real(cs.decay[n])
            self.curl[n] = c if cs.curl[n] is None else self.real(cs.curl[n])
        self.inv = {"e": [self.real(v) for v in cs.inv_e], "h": [self.real(v) for v in cs.inv_h]}
        self.cpml = {k: [self.real(v) for v in vs] for k, vs in cs.cpml.items()}
        self.masks = {n: self.edges(n) for n in E_CURL}
        self.poles = [dict(p=p, drive=self.real(p.drive), inv=self.real(p.inv_eps), P=0.0, J=0.0) for p in cs.poles]
        if cs.aux_line is not None:
            a = cs.aux_line
            self.line = {k: self.real(getattr(a, k)) for k in ("e_decay", "e_curl", "h_decay", "h_curl", "source")}
            self.line_e = torch.zeros_like(self.line["e_decay"])
            self.line_h = torch.zeros_like(self.line["h_decay"])
            self.line_patches = [(p, self.real(p.coeff),
                                  torch.as_tensor(np.asarray(p.sample_index, np.int64), device=DEVICE))
                                 for p in cs.line_patches]
        self.patches = [(p, self.real(p.coeff)) for p in cs.patches]
        self.shifted = [(p, self.real(p.scale), self.real(p.delay)) for p in cs.shifted]
        omega = 2.0 * np.pi * np.asarray(cs.frequencies, np.float64)
        self.omega = torch.as_tensor(omega, device=DEVICE)
        self.sums = [0.0] * len(cs.regions)

    @staticmethod
    def real(v):
        return torch.as_tensor(np.asarray(v), device=DEVICE).to(torch.float64)

    def edges(self, n):
        """(cells that keep their value, cells that are zeroed) of an E component on the outer faces."""
        shape = self.F[n].shape
        keep, wrap, pec = (torch.zeros(shape, dtype=torch.bool, device=DEVICE) for _ in range(3))
        for axis, _, _ in E_CURL[n]:
            for side in (0, 1):
                mode = self.cs.boundary[2 * axis + side]
                face = [slice(None)] * 3
                face[axis] = 0 if side == 0 else -1
                into = pec if mode == wm.BOUNDARY_PEC else (
                    wrap if mode in (wm.BOUNDARY_PERIODIC, wm.BOUNDARY_BLOCH) else keep)
                into[tuple(face)] = True
        return keep & ~wrap & ~pec, pec

    def stretch(self, d, n, axis, which):
        """CPML: psi = b psi + c d; d / kappa + psi."""
        if self.cs.pml_lo[axis] + self.cs.pml_hi[axis] == 0:
            return d
        b, c, ik = (_along(self.cpml["%s_%s" % (k, which)][axis][:d.shape[axis]], axis) for k in ("b", "c", "ik"))
        self.psi[n, axis] = b * self.psi.get((n, axis), 0.0) + c * d
        return ik * d + self.psi[n, axis]

    def backward_difference(self, f, axis):
        lo, hi = f.narrow(axis, 0, 1), f.narrow(axis, f.shape[axis] - 1, 1)
        if self.cs.boundary[2 * axis] in (wm.BOUNDARY_PERIODIC, wm.BOUNDARY_BLOCH):
            phase = complex(self.cs.bloch_cos[axis], self.cs.bloch_sin[axis])
            phase = phase if self.wave else phase.real
            lo, hi = hi * (phase.conjugate() if self.wave else phase), lo * phase
        return torch.diff(torch.cat([lo, f, hi], dim=axis), dim=axis) * _along(self.inv["e"][axis], axis)

    def add(self, name, box, value, channel=0):
        if channel:
            value = 1j * value
        grid = torch.zeros_like(self.F[name])
        grid[_box(box)] = value.to(self.kind)
        self.F[name] = self.F[name] + grid

    def line_terms(self, letter, values):
        for p, coeff, index in self.line_patches:
            if p.component[0] == letter:
                self.add(p.component, p.box, coeff * _along(values[index], p.sample_axis) * p.scale)

    def soft_terms(self, letter, n):
        for p, coeff in self.patches:
            if p.component[0] == letter:
                self.add(p.component, p.box, coeff * float(p.signal[n]), p.channel)
        for p, scale, delay in self.shifted:
            if p.component[0] == letter:
                st = p.source_time
                tau = n * self.cs.dt + p.t_offset - delay - st.resolved_delay
                wave = torch.exp(-0.5 * (tau * 2.0 * math.pi * st.fwidth) ** 2) * torch.cos(
                    2.0 * math.pi * st.frequency * tau + st.phase)
                self.add(p.component, p.box, scale * st.amplitude * wave, p.channel)

    def step(self, n):
        cs, F = self.cs, self.F
        for name, terms in H_CURL.items():
            curl = 0.0
            for axis, of, sign in terms:
                d = torch.diff(F[of], dim=axis) * _along(self.inv["h"][axis], axis)
                curl = curl + sign * self.stretch(d, name, axis, "h")
            F[name] = F[name] * self.decay[name] + self.curl[name] * curl
        if cs.aux_line is not None:
            self.line_terms("H", self.line_e)
            ln = self.line
            self.line_h = ln["h_decay"] * self.line_h - ln["h_curl"] * torch.diff(self.line_e)
        self.soft_terms("H", n)
        old = {name: F[name] for name in E_CURL}
        for name, terms in E_CURL.items():
            curl = 0.0
            for axis, of, sign in terms:
                curl = curl + sign * self.stretch(self.backward_difference(F[of], axis), name, axis, "e")
            keep, pec = self.masks[name]
            new = F[name] * self.decay[name] + self.curl[name] * curl
            F[name] = torch.where(keep, F[name], torch.where(pec, torch.zeros_like(new), new))
        if cs.aux_line is not None:
            self.line_terms("E", self.line_h)
            ln = self.line
            e = self.line_e.clone()
            e[1:-1] = ln["e_decay"][1:-1] * e[1:-1] - ln["e_curl"][1:-1] * torch.diff(self.line_h)
            e[0] = self.line_e[0]
            e[cs.aux_line.source_index] = ln["source"][n]
            e[-1] = 0.0
            self.line_e = e
        self.soft_terms("E", n)
        for q in self.poles:
            p = q["p"]
            e = old[p.component][_box(p.box)]
            if p.kind == 0:
                P = p.decay * q["P"] + q["drive"] * e
                q["J"] = (P - q["P"]) / cs.dt
                q["P"] = P
            else:
                q["J"] = p.decay * q["J"] - p.restoring * q["P"] + q["drive"] * e
                q["P"] = q["P"] + cs.dt * q["J"] if p.kind == 2 else 0.0
            self.add(p.component, p.box, -cs.dt * q["inv"] * q["J"])
        if cs.aux_line is None:
            for name in E_CURL:
                F[name] = F[name].masked_fill(self.masks[name][1], 0.0)
        for at, reg in enumerate(cs.regions):
            late = 0.0 if reg.component[0] == "E" else 0.5
            turn = torch.exp(1j * self.omega * ((n - late) * cs.dt)) * torch.as_tensor(cs.window[n], device=DEVICE)
            self.sums[at] = self.sums[at] + turn[:, None, None, None] * F[reg.component][_box(reg.box)][None]

    def spectra(self, steps):
        cs, out = self.cs, {}
        scale = 2.0 / np.sum(cs.window[:steps], axis=0)
        for reg, s in zip(cs.regions, self.sums):
            at = [cs.frequencies.index(f) for f in cs.monitor_frequencies[reg.monitor]]
            out.setdefault(reg.monitor, {})[reg.component] = s[at] * float(scale)
        return out


def _exact_design(case, seed):
    sc = _scene(case, np.random.default_rng([seed, 1]))
    eps = _design_eps(case, seed).double().requires_grad_(True)
    region = sc.material_regions[0]
    sc.material_regions = [dataclasses.replace(region, eps_r=eps.detach().cpu().numpy())]
    cs = wm.compile_scene(sc, case["steps"])
    dense = _Dense(cs)
    node = np.ones(cs.nodes)
    for st in sc.structures:
        node[st.geometry.node_mask(cs.nodes)] = st.medium.eps_r
    node = _Dense.real(node)
    node[tuple(slice(a, b) for a, b in zip(region.lo, region.hi))] = eps
    for axis, name in enumerate(E_CURL):
        pair = node.narrow(axis, 0, node.shape[axis] - 1) + node.narrow(axis, 1, node.shape[axis] - 1)
        dense.curl[name] = cs.dt / (0.5 * wm.scene.EPSILON_0 * pair)
    for n in range(case["steps"]):
        dense.step(n)
    spectra = dense.spectra(case["steps"])["patch"]
    loss = sum(v.abs().square().sum() for v in spectra.values())
    loss.backward()
    return {"spectra": {k: v.detach() for k, v in spectra.items()}, "grad": eps.grad}


def exact(case, seed):
    if case["kind"] == "design":
        # the saved history of larger ones does not fit
        return _exact_design(case, seed) if case["nx"] <= 80 else None
    results = []
    with torch.no_grad():
        for at, cs in enumerate(_compiled(case, seed)):
            dense = _Dense(cs)
            if case["kind"] != "solve":
                for name in COMPONENTS:
                    dense.F[name] = _field(cs, name, seed + 1000 * at).to(dense.kind)
            for n in range(case["steps"]):
                dense.step(n)
            out = {"spectra": dense.spectra(case["steps"])}
            if case["kind"] == "batch":
                out["spectra"] = torch.cat([v.reshape(-1) for m in out["spectra"].values() for v in m.values()])
            out["fields"] = {name: dense.F[name].real.contiguous() for name in COMPONENTS}
            if cs.complex_fields:
                out["imag"] = {name: dense.F[name].imag.contiguous() for name in COMPONENTS}
            results.append(out)
    return results if case["kind"] == "batch" else results[0]
