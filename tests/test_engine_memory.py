"""Where an engine's device memory comes from and goes back to: torch's caching
allocator for the solvers of this package, the device for engines that were created
through the C ABI without an allocator.  Nothing is held where neither can reach it."""
from __future__ import annotations

import ctypes
import gc
import subprocess
import sys

import pytest
import torch

from conftest import ROOT, load_package

pytestmark = pytest.mark.gpu
MIB = 1 << 20
FIELDS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


def _compiled(wm, n=160):
    return wm.compile_scene(wm.Scene(cells=(n,) * 3, spacing=25e-9, pml_cells=8), 4)


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_a_closed_solvers_memory_serves_the_next_tensors():
    wm = load_package()
    cs = _compiled(wm)
    wm.solver.B200FDTD(cs).init_field().close()  # the context and the kernels are loaded
    gc.collect()
    torch.cuda.empty_cache()
    before, held = _free(), torch.cuda.memory_allocated()
    solver = wm.solver.B200FDTD(cs).init_field()
    solver.step_range(0, 2)
    size = torch.cuda.memory_allocated() - held
    assert size > 12 * 4 * 160 ** 3  # both sets of the six fields, at least
    solver.close()
    assert torch.cuda.memory_allocated() == held
    # tensors of the fields' size take none from the device while the solver's lies there
    low = _free()
    tensors = [torch.empty(160 ** 3, device="cuda") for _ in range(12)]
    assert _free() >= low - 4 * MIB
    del tensors
    torch.cuda.empty_cache()
    assert _free() >= before - 4 * MIB


def _tfsf(wm, boundary):
    sc = wm.Scene(cells=(32, 28, 30), spacing=25e-9, pml_cells=6, boundary=boundary)
    sc.structures.append(wm.Structure(wm.Box((12, 11, 12), (18, 16, 17)), wm.Medium(eps_r=3.0)))
    sc.structures.append(wm.Structure(wm.Sphere((16.0, 14.0, 15.0), 3.0), wm.Medium.lorentz(2.0, 3.0, 250e12, 20e12)))
    pulse = wm.GaussianPulse(300e12, 100e12, delay=0.5e-15)
    if 2 in boundary or 3 in boundary:
        sc.sources.append(wm.PointDipole((14, 13, 14), "Ex", pulse, width=25e-9))
        if 3 in boundary:
            sc.bloch_k = (2e6, 1e6, 0.0)
    else:
        sc.sources.append(wm.PlaneWaveTFSF((1, 0, 0), (0, 0, 1), pulse, (9, 9, 9), (23, 19, 21)))
    sc.monitors.append(wm.PlaneMonitor("plane", 2, 15, frequencies=(250e12, 300e12)))
    return sc


@pytest.mark.parametrize("storage,boundary", [
    ("fp32", (1,) * 6), ("fp16", (1,) * 6), ("bf16", (1,) * 6), ("fp32", (4,) * 6), ("fp16", (4,) * 6),
    ("fp32", (2, 2, 2, 2, 1, 1)), ("fp32", (3, 3, 3, 3, 1, 1)),
])
def test_an_engine_reads_nothing_that_its_memory_held_before(storage, boundary, monkeypatch):
    """The same scales, fields and spectra on memory that holds 1.2e30 everywhere."""
    wm = load_package()
    held = {}

    @wm._lib.ALLOC_FN
    def alloc(nbytes, device, stream, user):
        t = torch.full((nbytes,), 0x71, dtype=torch.uint8, device="cuda")
        held[t.data_ptr()] = t
        return t.data_ptr()

    @wm._lib.FREE_FN
    def release(memory, user):
        del held[memory]

    cs = wm.compile_scene(_tfsf(wm, boundary), 40)
    runs = []
    for poisoned in (False, True):
        if poisoned:
            monkeypatch.setattr(wm.solver, "_torch_alloc", alloc)
            monkeypatch.setattr(wm.solver, "_torch_free", release)
        solver = wm.solver.B200FDTD(cs, storage=storage).init_field()
        assert bool(held) == poisoned
        scales = solver.storage_scales()
        solver.step_range(0, 40)
        fields = {n: solver.field(n) for n in FIELDS}
        spectra = {c: v.clone() for c, v in solver.monitor_results()["plane"].items()}
        solver.close()
        runs.append((scales, fields, spectra))
    assert not held
    assert runs[0][0] == runs[1][0]
    for k in (1, 2):
        for name, v in runs[0][k].items():
            assert torch.equal(v, runs[1][k][name]), name
    assert float(runs[0][1]["Ez"].abs().max()) > 0


@pytest.mark.parametrize("held", ["solver", "batch", "everything"])
def test_solvers_may_be_open_when_the_interpreter_ends(held):
    """Nothing is closed: the engines go with the modules whose functions free them."""
    code = f"""
import sys
sys.path.insert(0, {str(ROOT / "tests")!r})
from conftest import ROOT, load_package
wm = load_package()
cs = wm.compile_scene(wm.Scene(cells=(20, 20, 20), spacing=25e-9, pml_cells=4), 64)
solver = wm.solver.B200FDTD(cs).init_field()
solver.step_range(0, 4)
if {held!r} != "solver":
    batch = wm.solver.B200Batch([wm.solver.B200FDTD(cs) for _ in range(2)])
    batch.step_range(0, 40)
if {held!r} == "everything":
    sys.keep = [solver, batch]  # beyond the modules
    sys.keep.append(sys.keep)
print("stepped")
"""
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0 and done.stdout.split() == ["stepped"], (done.returncode, done.stderr[-2000:])


def test_an_engine_without_an_allocator_gives_its_memory_back_at_once():
    wm = load_package()
    lib = wm._lib.load()
    desc = wm._lib.FdtdGridDesc()
    desc.nx = desc.ny = desc.nz = 161
    desc.dt = 4e-17
    for f in range(6):
        desc.boundary[f] = 4
    free = []
    for _ in range(2):
        handle = ctypes.c_void_p()
        wm._lib.check(lib.fdtd_engine_create(ctypes.byref(desc), None, ctypes.byref(handle)), "create")
        inside = _free()
        wm._lib.check(lib.fdtd_engine_destroy(handle), "destroy")
        free.append(torch.cuda.mem_get_info()[0])
        assert free[-1] - inside > 12 * 4 * 160 ** 3 - 4 * MIB
    assert abs(free[1] - free[0]) <= 4 * MIB


def test_an_allocator_that_fails_is_an_error_and_leaves_nothing_behind():
    wm = load_package()
    lib = wm._lib.load()
    held = {}

    @wm._lib.ALLOC_FN
    def alloc(nbytes, device, stream, user):
        if len(held) == 7:
            return None
        t = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        held[t.data_ptr()] = t
        return t.data_ptr()

    @wm._lib.FREE_FN
    def release(memory, user):
        del held[memory]

    desc = wm._lib.FdtdGridDesc()
    desc.nx = desc.ny = desc.nz = 33
    desc.dt = 4e-17
    handle = ctypes.c_void_p()
    rc = lib.fdtd_engine_create_with(ctypes.byref(desc), None, alloc, release, None, ctypes.byref(handle))
    assert rc != 0 and not handle.value and not held
    assert b"out of memory" in lib.fdtd_last_error()
    only_one = lib.fdtd_engine_create_with(ctypes.byref(desc), None, alloc, wm._lib.FREE_FN(), None, ctypes.byref(handle))
    assert only_one == -1
