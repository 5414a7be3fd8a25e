"""Batched scenes (fdtd_batch_*): independent engines stepped together through
graph-captured step blocks give exactly the fields and monitor spectra of the
same engines stepped one by one (same kernels, same per-scene order)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu
FIELDS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


def _scenes(wm):
    return wm.workloads.batched_designs(n_scenes=4, seed=3, size_range=(24, 40), pml=4, n_freq=3)


def _state(solver):
    fields = {n: solver.field(n).cpu().numpy() for n in FIELDS}
    mons = {k: {c: v.cpu().numpy() for c, v in d.items()} for k, d in solver.monitor_results().items()}
    return fields, mons


def test_batch_equals_individual_runs():
    wm = load_package()
    steps = 70  # two graph blocks of 32 steps and a 6-step tail
    compiled = [wm.compile_scene(sc, steps) for sc in _scenes(wm)]
    ref = []
    for cs in compiled:
        s = wm.solver.B200FDTD(cs).init_field()
        # same call split as the batch below, so the monitor samples are
        # flushed into the DFT sums in the same groups
        s.step_range(0, 40)
        s.step_range(40, steps)
        ref.append(_state(s))
        s.close()
    solvers = [wm.solver.B200FDTD(cs).init_field() for cs in compiled]
    batch = wm.solver.B200Batch(solvers)
    batch.step_range(0, 40)
    batch.step_range(40, steps)
    info = batch.info()
    assert info["scenes"] == 4 and info["block_steps"] == 32 and info["graph_launches"] == 1
    for s, (rf, rm) in zip(solvers, ref):
        f, m = _state(s)
        for n in FIELDS:
            np.testing.assert_array_equal(f[n], rf[n])
        for mon, comps in rm.items():
            for c, v in comps.items():
                np.testing.assert_array_equal(m[mon][c], v)
    batch.close()
    for s in solvers:
        s.close()


def test_batch_autotune_keeps_results():
    wm = load_package()
    steps = 64
    compiled = [wm.compile_scene(sc, steps) for sc in _scenes(wm)[:2]]
    ref = []
    for cs in compiled:
        s = wm.solver.B200FDTD(cs).init_field()
        s.step_range(0, steps)
        ref.append(_state(s)[1])
        s.close()
    solvers = [wm.solver.B200FDTD(cs).init_field() for cs in compiled]
    batch = wm.solver.B200Batch(solvers)
    batch.autotune()  # picks launch shapes; the state is restored
    batch.step_range(0, steps)
    for s, rm in zip(solvers, ref):
        m = _state(s)[1]
        for mon, comps in rm.items():
            for c, v in comps.items():
                # another launch variant may contract a different multiply-add pair
                assert np.linalg.norm(m[mon][c] - v) <= 1e-5 * max(np.linalg.norm(v), 1e-30)
    batch.close()
    for s in solvers:
        s.close()


def _closed_scene(wm, cells, n_sources, steps, pml=0):
    sc = wm.Scene(cells=cells, spacing=25e-9, pml_cells=pml, boundary=(1,) * 6 if pml else (4,) * 6)
    for n in range(n_sources):
        at = (3 + n % 5 * 3, 4 + n // 5 * 3, cells[2] // 2)
        sc.sources.append(wm.PointDipole(at, "Ez", wm.GaussianPulse(300e12, 100e12, delay=0.5e-15), width=25e-9))
    sc.monitors.append(wm.PointMonitor("probe", tuple(c // 2 for c in cells), frequencies=(250e12, 300e12)))
    return wm.compile_scene(sc, steps)


def test_batch_autotune_gives_equal_scenes_the_same_launch():
    """Engines of one shape take the tuned tile as it is, its rows included."""
    wm = load_package()
    solvers = [wm.solver.B200FDTD(_closed_scene(wm, (96, 96, 96), 1, 64, pml=8)).init_field() for _ in range(3)]
    batch = wm.solver.B200Batch(solvers)
    batch.autotune()
    launches = [s.get_launch() for s in solvers]
    assert launches[0][0] == 11 and launches[0][1] > 1
    assert launches == [launches[0]] * 3
    batch.close()
    for s in solvers:
        s.close()


@pytest.mark.parametrize("shapes", [
    [((20, 20, 24), 24), ((20, 20, 24), 25)],    # one size class: 24 injection terms, and more than the quad tile takes
    [((20, 20, 511), 1), ((20, 20, 512), 1)],    # 512 z nodes, and one more
    [((20, 30, 40), 1), ((21, 24, 42), 1)],      # other row lengths and counts
])
def test_batch_autotune_of_a_mixed_class(shapes):
    wm = load_package()
    steps = 32
    compiled = [_closed_scene(wm, cells, n, steps) for cells, n in shapes]
    ref = []
    for cs in compiled:
        s = wm.solver.B200FDTD(cs).init_field()
        s.step_range(0, steps)
        ref.append(_state(s))
        s.close()
    solvers = [wm.solver.B200FDTD(cs).init_field() for cs in compiled]
    batch = wm.solver.B200Batch(solvers)
    batch.autotune()
    batch.step_range(0, steps)
    for s, (rf, _) in zip(solvers, ref):
        f, _ = _state(s)
        for group in (FIELDS[:3], FIELDS[3:]):
            # another kernel rounds up to three products of a cell differently each step (Hz
            # of z dipoles is nothing but such rounding: E and H as wholes)
            got, want = (np.concatenate([x[n].ravel() for n in group]).astype(np.float64) for x in (f, rf))
            assert np.linalg.norm(want) > 0
            assert np.linalg.norm(got - want) <= 3 * steps * 2.0 ** -24 * np.linalg.norm(want)
    batch.close()
    for s in solvers:
        s.close()


def test_batch_rejects_mismatched_sample_blocks():
    wm = load_package()
    compiled = [wm.compile_scene(sc, 10) for sc in _scenes(wm)[:2]]
    a = wm.solver.B200FDTD(compiled[0]).init_field()
    b = wm.solver.B200FDTD(compiled[1], sample_block=16).init_field()
    with pytest.raises(wm._lib.FdtdError):
        wm.solver.B200Batch([a, b])
    a.close()
    b.close()


def test_batch_adjoint_equals_individual_problems():
    """Per-scene adjoint gradients of a batched forward run (checkpoints every 40
    steps, graph-captured batch steps) equal one DesignProblem per scene."""
    wm = load_package()
    adj = wm.adjoint
    steps, stride = 120, 40
    scenes = wm.workloads.batched_designs(n_scenes=3, seed=5, size_range=(36, 44), pml=4, n_freq=3, design=True)
    eps = [sc.material_regions[0].eps_r for sc in scenes]

    def seeds(mons):
        return {"probe": {c: 2.0 * v for c, v in mons["probe"].items()}}

    ref = []
    for sc, e in zip(scenes, eps):
        p = adj.DesignProblem(sc, steps, stride=stride, history="replay")
        ref.append((p.forward(e), None))
        ref[-1] = (ref[-1][0], p.backward(seeds(ref[-1][0])))
        p.close()
    batch = adj.BatchDesignProblem(scenes, steps, stride=stride)
    mons = batch.forward(eps)
    grads = batch.backward([seeds(m) for m in mons])
    assert set(batch.timings) == {"forward_ms", "backward_ms"}
    for (rm, rg), m, g in zip(ref, mons, grads):
        for c, v in rm["probe"].items():
            np.testing.assert_allclose(m["probe"][c].cpu().numpy(), v.cpu().numpy(), rtol=1e-6, atol=0)
        assert np.abs(rg).max() > 0
        np.testing.assert_allclose(g, rg, rtol=1e-5, atol=1e-6 * np.abs(rg).max())
    batch.close()
