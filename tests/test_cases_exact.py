"""Small scenes of the kinds that perf/cases.py steps, against its dense 64-bit
restatement with its tolerances: closed, absorbing and graded grids, poles with a TFSF
plane wave, a Bloch grating with poles and its pulsed slab (complex field), a batch, and
a design's gradient."""
from __future__ import annotations

import importlib.util
import sys

import pytest
import torch

from conftest import ROOT, load_package

pytestmark = pytest.mark.gpu


def _cases():
    load_package()  # under the name by which the cases look for it
    if "perf_cases" not in sys.modules:
        spec = importlib.util.spec_from_file_location("perf_cases", ROOT / "perf" / "cases.py")
        module = importlib.util.module_from_spec(spec)
        sys.modules["perf_cases"] = module
        spec.loader.exec_module(module)
    return sys.modules["perf_cases"]


def _flat(out, path=""):
    if isinstance(out, dict):
        out = out.items()
    elif isinstance(out, (list, tuple)):
        out = enumerate(out)
    else:
        return {path: torch.as_tensor(out)}
    return {k: v for key, value in out for k, v in _flat(value, f"{path}/{key}").items()}


@pytest.mark.parametrize("case", [
    dict(kind="steps", scene="cavity", nx=31, ny=26, nz=29, pml=0, steps=40, storage="fp32"),
    dict(kind="steps", scene="dielectric", nx=37, ny=34, nz=38, pml=6, steps=40, storage="fp32"),
    dict(kind="steps", scene="graded", nx=35, ny=41, nz=30, pml=6, steps=40, storage="fp32"),
    dict(kind="steps", scene="dispersive", nx=52, ny=52, nz=52, pml=6, steps=30, storage="fp32"),
    dict(kind="steps", scene="grating", nx=64, ny=50, nz=112, pml=16, steps=24, storage="fp32"),
    dict(kind="batch", scene="designs", nx=72, ny=72, nz=72, pml=8, steps=40, scenes=3, storage="fp32"),
    dict(kind="design", scene="design", nx=80, ny=80, nz=48, pml=10, steps=120, stride=0, storage="fp32"),
], ids=lambda c: c["scene"])
def test_small_cases_against_64_bits(case):
    cases = _cases()
    seed = 7
    state = cases.prepare(case, seed)
    got = _flat(cases.run(state))
    want = _flat(cases.exact(case, seed))
    for solver in state.get("solvers", []):
        solver.close()
    tol = cases.tolerance(case)["rel"]
    assert got.keys() == want.keys()
    for path, exact in want.items():
        exact = exact.to(got[path].device)
        norm = float(torch.linalg.vector_norm(exact))
        assert norm > 0, path
        # A spectrum is twice a weighted mean of field samples, so it is off by up to twice
        # as much as they are: by a share of their size, which that of one cell where
        # they cancel can lie far below.
        field = want.get("/0/fields/" + path.split("/")[-1], want.get("/fields/" + path.split("/")[-1]))
        if field is not None:
            norm = max(norm, 2.0 * (exact.numel() / field.numel()) ** 0.5 * float(torch.linalg.vector_norm(field)))
        assert float(torch.linalg.vector_norm(got[path] - exact)) <= tol * norm, path
