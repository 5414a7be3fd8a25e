"""The quad-tile step kernel (launch variant 11) at the edges of its tiles: ragged
row counts, z rows of every remainder mod 4 and of the longest length it takes,
one-plane chunks, slabs thinner and thicker than a quad, PEC and periodic faces,
poles, TFSF and point sources.

Every tile shape gives the same bits.  Against the warp kernel (variant 2) each
step differs by the rounding of at most three products per cell (2^-24 each), which
add up at most linearly: 3 * 40 steps * 6e-8 = 7e-6 of the field's norm.
"""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu
FIELDS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
STEPS = 40
TOL = 7e-6


def _scene(wm, cells, pml, boundary, tfsf=False):
    sc = wm.Scene(cells=cells, spacing=25e-9, pml_cells=pml, boundary=boundary)
    mid = tuple(c // 2 for c in cells)
    sc.structures.append(wm.Structure(wm.Box(tuple(m - 2 for m in mid), tuple(m + 3 for m in mid)), wm.Medium(eps_r=3.0)))
    sc.structures.append(wm.Structure(wm.Sphere(tuple(float(m) for m in mid), 2.4), wm.Medium.lorentz(2.0, 3.0, 250e12, 20e12)))
    pulse = wm.GaussianPulse(300e12, 100e12, delay=0.5e-15)
    if tfsf:
        sc.sources.append(wm.PlaneWaveTFSF((1, 0, 0), (0, 0, 1), pulse, (pml + 2,) * 3, tuple(c - pml - 2 for c in cells)))
    else:
        sc.sources.append(wm.PointDipole(mid, "Ez", pulse, width=25e-9))
    return wm.compile_scene(sc, STEPS)


def _run(wm, cs, launch):
    solver = wm.solver.B200FDTD(cs).init_field()
    if launch is not None:
        solver.set_launch(*launch)
    variant = solver.get_launch()[0]
    solver.step_range(0, STEPS)
    out = {n: solver.field(n).cpu().numpy() for n in FIELDS}
    solver.close()
    return variant, out


@pytest.mark.parametrize("cells,pml,boundary,tfsf", [
    ((17, 13, 12), 3, (1,) * 6, False),      # one cell beyond whole quads, thin slabs
    ((16, 14, 15), 5, (1,) * 6, False),      # whole quads, slabs across quads
    ((21, 30, 34), 6, (1,) * 6, True),       # TFSF faces on every axis
    ((12, 11, 13), 0, (4,) * 6, False),      # closed box
    ((14, 12, 29), 4, (2, 2, 2, 2, 1, 1), False),   # periodic x, y with z slabs and poles
    ((14, 12, 18), 4, (4, 4, 2, 2, 1, 4), False),   # PEC beside periodic faces
    ((9, 8, 511), 3, (1,) * 6, False),       # the longest row
])
def test_tiles_agree_with_each_other_and_with_the_warp_kernel(cells, pml, boundary, tfsf):
    wm = load_package()
    cs = _scene(wm, cells, min(pml, (min(cells) - 2) // 2), boundary, tfsf)
    variant, base = _run(wm, cs, None)
    assert variant == 11
    top = 3 if cells[2] > 256 else 9
    for tile in ((11, 1, 1), (11, top, 5), (11, 2, cells[0] + 1)):
        _, got = _run(wm, cs, tile)
        for n in FIELDS:
            np.testing.assert_array_equal(got[n], base[n], err_msg=f"{tile} {n}")
    _, ref = _run(wm, cs, (2, 1, 0))
    num = sum(np.linalg.norm(base[n].astype(np.float64) - ref[n]) ** 2 / np.linalg.norm(ref[n].astype(np.float64)) ** 2 for n in FIELDS)
    assert np.sqrt(num) <= TOL


@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 6, 7])
def test_lanes_past_the_last_quad_leave_the_fields_alone(rows):
    """Tiles whose (rows + 1) * 6 quads end inside a warp: the lanes past the last quad
    repeat it and may write nothing.  TFSF faces put H terms (added to the H that the
    ring holds) on rows of every place in a tile, the last one among them."""
    wm = load_package()
    cs = _scene(wm, (13, 14, 22), 2, (1,) * 6, tfsf=True)
    assert (rows + 1) * ((cs.nodes[2] + 3) // 4) % 32 != 0
    _, one = _run(wm, cs, (11, 15, 3))
    _, got = _run(wm, cs, (11, rows, 4))
    _, ref = _run(wm, cs, (2, 1, 0))
    for n in FIELDS:
        np.testing.assert_array_equal(got[n], one[n], err_msg=n)
        assert np.linalg.norm(ref[n]) > 0
    num = sum(np.linalg.norm(got[n].astype(np.float64) - ref[n]) ** 2 / np.linalg.norm(ref[n].astype(np.float64)) ** 2 for n in FIELDS)
    assert np.sqrt(num) <= TOL


@pytest.mark.parametrize("pml,boundary,other", [(0, (4,) * 6, 10), (3, (1,) * 6, 2), (3, (2, 2, 2, 2, 1, 1), 2)])
def test_terms_beyond_the_table_run_another_kernel(pml, boundary, other):
    """24 injection terms fit the kernel's table; with 25 the engine runs the kernel that
    it would run without this one."""
    wm = load_package()
    for n_terms, variant in ((24, 11), (25, other)):
        sc = wm.Scene(cells=(18, 17, 19), spacing=25e-9, pml_cells=pml, boundary=boundary)
        for n in range(n_terms):
            pulse = wm.GaussianPulse(300e12, 100e12, delay=0.5e-15)
            sc.sources.append(wm.PointDipole((4 + n % 5 * 2, 4 + n // 5 * 2, 8), "E" + "xyz"[n % 3], pulse, width=25e-9))
        cs = wm.compile_scene(sc, STEPS)
        picked, got = _run(wm, cs, None)
        assert picked == variant
        _, ref = _run(wm, cs, (2, 1, 0))
        num = sum(np.linalg.norm(got[n].astype(np.float64) - ref[n]) ** 2 / np.linalg.norm(ref[n].astype(np.float64)) ** 2 for n in FIELDS)
        assert np.sqrt(num) <= TOL


def test_many_terms_on_a_row_shorten_the_chunks():
    """Sources over the same cells of a closed box: shorter chunks (a CTA that holds them
    all ends last) and the fields of the longer ones; a launch that is set stays."""
    wm = load_package()
    launches, fields = [], []
    for n_terms, launch in ((1, None), (12, None), (12, (11, 0, 40))):
        sc = wm.Scene(cells=(120, 64, 64), spacing=25e-9, boundary=(4,) * 6)
        for n in range(n_terms):
            pulse = wm.GaussianPulse(300e12, 100e12, delay=0.5e-15)
            sc.sources.append(wm.PointDipole((60 + n % 3, 32 + n // 3, 32), "E" + "xyz"[n % 3], pulse, width=25e-9))
        solver = wm.solver.B200FDTD(wm.compile_scene(sc, STEPS)).init_field()
        if launch:
            solver.set_launch(*launch)
        launches.append(solver.get_launch())
        solver.step_range(0, STEPS)
        fields.append({n: solver.field(n).cpu().numpy() for n in FIELDS})
        solver.close()
    assert launches[0][0] == launches[1][0] == 11 and launches[2][2] == 40
    assert launches[1][2] < launches[0][2]
    for n in FIELDS:
        np.testing.assert_array_equal(fields[1][n], fields[2][n])


def test_poles_in_the_step_kernel_run_the_warp_kernels_launch():
    """Without the ADE pass the warp kernel runs, on its own chunks; with it again, the
    quad tile as before.  A launch that was set stays."""
    wm = load_package()
    cs = _scene(wm, (60, 50, 40), 4, (1,) * 6)
    solver = wm.solver.B200FDTD(cs).init_field()
    first = solver.get_launch()
    solver.set_ade_pass(False)
    off = solver.get_launch()
    solver.step_range(0, 4)
    solver.set_ade_pass(True)
    assert solver.get_launch() == first
    solver.set_launch(2, 0, 0)
    assert off == (11,) + solver.get_launch()[1:]
    solver.set_launch(11, 3, 7)
    solver.set_ade_pass(False)
    assert solver.get_launch() == (11, 3, 7)
    solver.close()


def test_rows_beyond_a_tile_run_another_kernel():
    wm = load_package()
    solver = wm.solver.B200FDTD(_scene(wm, (8, 8, 512), 2, (1,) * 6)).init_field()
    assert solver.get_launch()[0] == 2
    with pytest.raises(wm._lib.FdtdError):
        solver.set_launch(11, 0, 0)
    solver.step_range(0, 4)
    solver.close()


def test_two_threads_step_tiles_of_different_sizes():
    """Two solvers of one kernel, one on the largest tile and one on the smallest, stepped
    on a stream and a thread each: neither makes the other's launch fail, and both give
    the fields of stepping alone."""
    import threading

    import torch

    wm = load_package()
    cases = [((12, 40, 120), (11, 18, 13)), ((12, 9, 10), (11, 1, 13))]  # 190 and 3 KB of shared memory
    scenes = [_scene(wm, cells, 3, (1,) * 6) for cells, _ in cases]
    want = [_run(wm, cs, launch)[1] for cs, (_, launch) in zip(scenes, cases)]
    got, errors = [None, None], []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                solver = wm.solver.B200FDTD(scenes[k]).init_field()
                solver.set_launch(*cases[k][1])
                solver.checkpoint_save(0)
                start.wait()
                for _ in range(400):
                    solver.checkpoint_load(0)
                    solver.step_range(0, STEPS)
                got[k] = {n: solver.field(n).cpu().numpy() for n in FIELDS}
                solver.close()
        except Exception as err:  # noqa: BLE001 (reported below)
            errors.append(err)

    start = threading.Barrier(2, timeout=60)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for k in range(2):
        for n in FIELDS:
            np.testing.assert_array_equal(got[k][n], want[k][n])


def test_a_wait_that_runs_out_is_reported():
    wm = load_package()
    solver = wm.solver.B200FDTD(_scene(wm, (24, 20, 18), 4, (1,) * 6)).init_field()
    solver.set_wait_limit(0)
    with pytest.raises(wm._lib.FdtdError) as err:
        solver.step_range(0, 2)
    assert "status -5" in str(err.value)
    solver.set_wait_limit(1 << 20)
    solver.step_range(2, 4)
    solver.close()


@pytest.mark.parametrize("bloch", [False, True])
def test_spectra_equal_the_scaled_accumulators(bloch):
    """monitor_results against raw_dft, scaled here: the same products, so the same
    bits.  Monitors of other frequencies, a one-cell monitor and a whole plane."""
    import torch

    wm = load_package()
    sc = wm.Scene(cells=(18, 14, 20), spacing=25e-9, pml_cells=4, boundary=(3, 3, 2, 2, 1, 1) if bloch else (1,) * 6,
                  bloch_k=(2e6, 0.0, 0.0) if bloch else (0.0, 0.0, 0.0))
    sc.sources.append(wm.PointDipole((9, 7, 10), "Ex", wm.GaussianPulse(300e12, 100e12, delay=0.5e-15), width=25e-9))
    sc.monitors.append(wm.PlaneMonitor("plane", 2, 8, frequencies=(250e12, 300e12, 350e12)))
    sc.monitors.append(wm.PointMonitor("point", (8, 6, 9), frequencies=(350e12, 250e12)))
    cs = wm.compile_scene(sc, STEPS)
    solver = wm.solver.B200FDTD(cs).init_field()
    solver.step_range(0, STEPS)
    got, host = solver.monitor_results(), solver.monitor_results(host=True)
    re, im = solver.raw_dft()
    if bloch:
        rb, ib = solver.raw_dft(imag=True)
        re, im = re - ib, im + rb
    scale = wm.scene.window_scales(cs.window, STEPS, len(cs.frequencies)).astype(np.float32)
    for reg, base in zip(cs.regions, solver.region_base):
        b = reg.box
        shape = (b[1] - b[0], b[3] - b[2], b[5] - b[4])
        for n, f in enumerate(cs.monitor_frequencies[reg.monitor]):
            at = cs.frequencies.index(f)
            want = torch.complex(re[at] * float(scale[at]), im[at] * float(scale[at]))[base:base + int(np.prod(shape))]
            v = got[reg.monitor][reg.component][n]
            assert torch.equal(v, want.reshape(shape))
            assert torch.equal(host[reg.monitor][reg.component][n], v.cpu())
    solver.close()


def test_released_memory_goes_back_to_the_device():
    """A closed solver's arrays stay with torch's allocator (a second one of the same
    scene takes them from there) until they are given back."""
    import torch

    wm = load_package()
    cs = wm.compile_scene(wm.Scene(cells=(96, 96, 96), spacing=25e-9, pml_cells=8), 4)
    wm.solver.release_memory()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        solver = wm.solver.B200FDTD(cs).init_field()
        solver.step_range(0, 2)
        assert float(solver.field("Ez").abs().max()) == 0.0  # reused memory starts at zero too
        solver.set_field("Ez", torch.ones(wm.scene.component_shape("Ez", cs.nodes), device="cuda"))
        solver.close()
    wm.solver.release_memory()
    assert torch.cuda.mem_get_info()[0] >= free - (64 << 20)  # torch's own cache: three 3.5 MB fields
