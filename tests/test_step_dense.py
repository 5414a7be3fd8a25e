"""One step forward and one step back of every cell against a dense 64-bit
restatement and its derivative (torch.autograd), on graded and uniform grids whose
slabs and faces end at every remainder of four z cells: the quad-tile kernel without
constant spacing, and the adjoint passes' four-cell box, its shell and grids too thin
for a box.

A value is the sum of at most 13 products (four differences, each over kappa and into
psi, and the value before), of three FP32 roundings each: 39 * 2^-24 = 2.3e-6 of an
array's largest value.
"""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest
import torch

from conftest import load_package

pytestmark = pytest.mark.gpu
TOL = 2.4e-6
E_NAMES, H_NAMES = ("Ex", "Ey", "Ez"), ("Hx", "Hy", "Hz")
FIELDS = E_NAMES + H_NAMES
# component -> ((axis, field, sign) of its curl terms, in the order of their psi)
H_CURL = {"Hx": ((1, "Ez", -1), (2, "Ey", 1)), "Hy": ((0, "Ez", 1), (2, "Ex", -1)), "Hz": ((0, "Ey", -1), (1, "Ex", 1))}
E_CURL = {"Ex": ((1, "Hz", 1), (2, "Hy", -1)), "Ey": ((0, "Hz", -1), (2, "Hx", 1)), "Ez": ((0, "Hy", 1), (1, "Hx", -1))}
P, E, N = 1, 4, 0


def _compiled(wm, cells, pml, boundary, graded):
    sc = wm.Scene(cells=cells, spacing=25e-9, pml_cells=pml, boundary=boundary)
    mid = tuple(c // 2 for c in cells)
    sc.structures.append(wm.Structure(wm.Box(tuple(m - 2 for m in mid), tuple(m + 2 for m in mid)), wm.Medium(eps_r=3.0)))
    cs = wm.compile_scene(sc, 4)
    if not graded:
        return cs
    inv_e, inv_h = [], []
    for a, n in enumerate(cs.nodes):
        node = 1.0 + 0.3 * np.linspace(-1.0, 1.0 + 0.1 * a, n) ** 2
        inv_e.append((float(cs.inv_e[a][0]) / node).astype(np.float32))
        inv_h.append((float(cs.inv_h[a][0]) / (0.5 * (node[1:] + node[:-1]))).astype(np.float32))
    return dataclasses.replace(cs, inv_e=inv_e, inv_h=inv_h)


def _along(values, axis):
    shape = [1, 1, 1]
    shape[axis] = -1
    return torch.as_tensor(np.asarray(values, np.float64)).reshape(shape)


def _slab(cs, axis, extent):
    """Cells of an axis that lie in its CPML slabs, in the order of a psi array."""
    return torch.tensor([*range(cs.pml_lo[axis]), *range(extent - cs.pml_hi[axis], extent)])


def _states(wm, cs):
    """Shapes of the state: ("f", component, 0) fields, ("p", component, term) psi."""
    shapes = {}
    for comp, name in enumerate(FIELDS):
        ext = wm.scene.component_shape(name, cs.nodes)
        shapes["f", comp, 0] = tuple(ext)
        for which, (axis, _, _) in enumerate((E_CURL if comp < 3 else H_CURL)[name]):
            if cs.pml_lo[axis] + cs.pml_hi[axis]:
                shapes["p", comp, which] = tuple(len(_slab(cs, axis, n)) if a == axis else n for a, n in enumerate(ext))
    return shapes


def _step(cs, x):
    """The next state, as torch expressions of the state x."""
    out = {}
    F = {name: x["f", comp, 0] for comp, name in enumerate(FIELDS)}

    def stretched(d, comp, which, axis, updated):
        key = ("p", comp, which)
        if key not in x:
            return d
        letter = "e" if comp < 3 else "h"
        cells = _slab(cs, axis, d.shape[axis])
        b, c, ik = (_along(cs.cpml[f"{k}_{letter}"][axis], axis).index_select(axis, cells) for k in ("b", "c", "ik"))
        at = d.index_select(axis, cells)
        psi = b * x[key] + c * at
        out[key] = torch.where(updated.index_select(axis, cells), psi, x[key])
        return d.index_copy(axis, cells, ik * at + psi)

    def advanced(name, curl):
        decay, scale = cs.uniform[name]
        decay = decay if cs.decay[name] is None else torch.as_tensor(np.asarray(cs.decay[name], np.float64))
        scale = scale if cs.curl[name] is None else torch.as_tensor(np.asarray(cs.curl[name], np.float64))
        return F[name] * decay + scale * curl

    new = {}
    for name, terms in H_CURL.items():
        comp = FIELDS.index(name)
        every = torch.ones(F[name].shape, dtype=torch.bool)
        curl = sum(sign * stretched(torch.diff(F[of], dim=axis) * _along(cs.inv_h[axis], axis), comp, which, axis, every)
                   for which, (axis, of, sign) in enumerate(terms))
        new[name] = advanced(name, curl)
    F.update(new)
    for name, terms in E_CURL.items():
        comp = FIELDS.index(name)
        keep, pec = (torch.zeros(F[name].shape, dtype=torch.bool) for _ in range(2))
        for axis, _, _ in terms:
            for side in (0, 1):
                face = pec if cs.boundary[2 * axis + side] == E else keep
                face.select(axis, 0 if side == 0 else face.shape[axis] - 1).fill_(True)
        curl = 0.0
        for which, (axis, of, sign) in enumerate(terms):
            pad = torch.zeros_like(F[of].narrow(axis, 0, 1))
            d = torch.diff(torch.cat([pad, F[of], pad], dim=axis), dim=axis) * _along(cs.inv_e[axis], axis)
            curl = curl + sign * stretched(d, comp, which, axis, ~keep & ~pec)
        new[name] = torch.where(pec, 0.0, torch.where(keep, F[name], advanced(name, curl)))
    for comp, name in enumerate(FIELDS):
        out["f", comp, 0] = new[name]
    return out


def _close(got, want, what):
    want = want.detach().numpy()
    assert np.abs(got - want).max() <= TOL * np.abs(want).max(), (what, np.unravel_index(np.abs(got - want).argmax(), want.shape))


@pytest.mark.parametrize("graded", [False, True])
@pytest.mark.parametrize("cells,pml,boundary", [
    ((13, 12, 11), 3, (P,) * 6),          # a box of one z quad
    ((16, 15, 17), 4, (P,) * 6),          # box from the slab's own end, two cells short of the other
    ((15, 17, 22), 5, (P,) * 6),          # slabs across quads
    ((14, 14, 14), 5, (P,) * 6),          # no whole z quad inside: no box
    ((24, 9, 21), 4, (P,) * 6),           # one row for the first pass, none for the second
    ((12, 13, 10), 0, (E,) * 6),          # no slab
    ((15, 14, 19), 4, (P, E, N, P, P, E)),
])
def test_a_step_and_its_transpose_cell_by_cell(cells, pml, boundary, graded):
    wm = load_package()
    lib = wm._lib.load()
    cs = _compiled(wm, cells, pml, boundary, graded)
    rng = np.random.default_rng(5)
    shapes = _states(wm, cs)
    # H in units of E over the vacuum impedance, psi in those of the other field a length
    field = {True: 1.0, False: 1.0 / 377.0}
    scale = {k: field[k[1] < 3] if k[0] == "f" else field[k[1] >= 3] / 25e-9 for k in shapes}
    x = {k: torch.tensor(scale[k] * rng.standard_normal(s), dtype=torch.float32) for k, s in shapes.items()}
    y = {k: torch.tensor(rng.standard_normal(s) / scale[k], dtype=torch.float32) for k, s in shapes.items()}
    at = {k: v.double().requires_grad_(True) for k, v in x.items()}
    want = _step(cs, at)
    back = torch.autograd.grad(sum((want[k] * y[k].double()).sum() for k in shapes), [at[k] for k in shapes])

    solver = wm.solver.B200FDTD(cs).init_field()
    h = solver.handle
    assert solver.get_launch()[0] == 11
    wm._lib.check(lib.fdtd_engine_adjoint_init(h, None, 1), "adjoint_init")
    code = {"f": 0, "p": 1}
    for (kind, comp, which), t in x.items():
        t = t.to(solver.device)
        if kind == "f":
            wm._lib.check(lib.fdtd_engine_pack_field(h, comp, wm._lib.ptr(t)), "pack")
        else:
            wm._lib.check(lib.fdtd_engine_pack_psi(h, comp, which, wm._lib.ptr(t)), "pack_psi")
        torch.cuda.synchronize()
    solver.step_range(0, 1)
    for (kind, comp, which), t in y.items():
        t = t.to(solver.device)
        wm._lib.check(lib.fdtd_engine_adjoint_pack(h, code[kind], comp, which, wm._lib.ptr(t)), "adj_pack")
        torch.cuda.synchronize()
    got = {}
    for kind, comp, which in shapes:
        t = torch.empty(shapes[kind, comp, which], device=solver.device)
        if kind == "f":
            wm._lib.check(lib.fdtd_engine_unpack_field(h, comp, wm._lib.ptr(t)), "unpack")
        else:
            wm._lib.check(lib.fdtd_engine_unpack_psi(h, comp, which, wm._lib.ptr(t)), "unpack_psi")
        got[kind, comp, which] = t.cpu().numpy()
    for k in shapes:
        _close(got[k], want[k], ("forward", k))
    wm._lib.check(lib.fdtd_engine_adjoint_range(h, 1, 0), "adjoint_range")
    for k, g in zip(shapes, back):
        t = torch.empty(shapes[k], device=solver.device)
        wm._lib.check(lib.fdtd_engine_adjoint_unpack(h, code[k[0]], k[1], k[2], wm._lib.ptr(t)), "adj_unpack")
        _close(t.cpu().numpy(), g, ("transpose", k))
    solver.close()
