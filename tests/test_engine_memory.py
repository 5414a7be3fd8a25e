"""Where an engine's device memory comes from and goes back to: torch's caching
allocator for the solvers of this package, the device for engines that were created
through the C ABI without an allocator.  Nothing is held where neither can reach it."""
from __future__ import annotations

import ctypes
import gc

import pytest
import torch

from conftest import load_package

pytestmark = pytest.mark.gpu
MIB = 1 << 20


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
    desc.nx = desc.ny = desc.nz = 17
    desc.dt = 4e-17
    handle = ctypes.c_void_p()
    rc = lib.fdtd_engine_create_with(ctypes.byref(desc), None, alloc, release, None, ctypes.byref(handle))
    assert rc != 0 and not handle.value and not held
    assert b"out of memory" in lib.fdtd_last_error()
    only_one = lib.fdtd_engine_create_with(ctypes.byref(desc), None, alloc, wm._lib.FREE_FN(), None, ctypes.byref(handle))
    assert only_one == -1
