"""The kernels that replaced plain ones, at the sizes where their own rules change:
the implicit and u2p passes around the warp's cell counts, the init's columns with
spin, the ordered folds around the chunk size, the ghost fill on every kind of
boundary; all bit for bit against the oracle."""
import ctypes
import subprocess

import numpy as np
import pytest

from tests.engine import koralcuda
from tests.orcsim import OracleSim
from tests.test_lean_solve import cells, lean_binary  # noqa: F401 (fixtures)

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, dtype=np.float64).view(np.uint64)


def _pair(nx, ny, nz, **opt):
    kc = koralcuda()
    kc.lib()
    grid, o = kc.puffy_grid(nx, ny, nz), kc.puffy_options(**opt)
    gpu, orc = kc.Sim(grid, o), OracleSim(grid, o, nthreads=8)
    assert gpu.initPuffy(1e-3, 1e-3, 5) == orc.init_puffy(1e-3, 1e-3, 5)
    orc.lib.orc_sim_init_timestep_guess(orc.h)
    return gpu, orc


def _same(gpu, orc):
    assert np.array_equal(_bits(gpu.p), _bits(orc.prims()))
    assert np.array_equal(_bits(gpu.u), _bits(orc.cons()))
    assert np.array_equal(gpu.flags, orc.flags())


@pytest.mark.parametrize("spin", [0.0, 0.5])
def test_init_columns_with_spin(spin):
    """The column solve with its angular momentum's powers multiplied away
    (no spin) and formed (spin); 43 x 37 columns are no multiple of a block's."""
    gpu, orc = _pair(43, 37, 1, bhspin=spin)
    _same(gpu, orc)


@pytest.mark.parametrize("shape", [(31, 21, 1), (37, 33, 1), (148, 9, 1), (149, 33, 4), (11, 13, 7)])
def test_steps_at_the_edges_of_the_solve_launches(shape):
    """651 and 1221 cells (2 and 4 cells a warp), few theta rows, 19668 cells
    (full warps, the last one partly filled), and a small grid with faces in
    all three directions (the update's streaming passes by component)."""
    gpu, orc = _pair(*shape)
    for _ in range(2):
        gpu.step()
        orc.step()
        _same(gpu, orc)


@pytest.mark.parametrize("opt", [{"radimp_start_with_bisect": 0}, {"radimp_scale_jacobian": 0}, {"radimp_lag_opac": 1},
                                 {"radimp_allow_rad_ceiling": 0, "radimp_allow_entr_in_4dprim": 0},
                                 {"radimp_opdamp_maxlevels": 1, "radimp_maxiter": 6}, {"synchrotron_bridge": 1}])
def test_implicit_options(opt):
    gpu, orc = _pair(32, 30, 1, **opt)
    for _ in range(2):
        gpu.step()
        orc.step()
        _same(gpu, orc)


@pytest.mark.parametrize("nz", [1, 5])
@pytest.mark.parametrize("bc", [(2, 2), (1, 2), (0, 1), (1, 0), (0, 0), (2, 1)])
def test_ghost_fill_on_every_boundary(bc, nz):
    """Faces and corners with periodic (0), copied (1) and PUFFY (2) x and y
    boundaries, in 2D (whose corner means look across a period) and in 3D."""
    gpu, orc = _pair(24, 20, nz, bc_x=bc[0], bc_y=bc[1], bc_z=0 if nz > 1 else 1)
    gpu.setBc()
    assert orc.lib.orc_sim_set_bc(orc.h) == 0
    _same(gpu, orc)


@pytest.mark.parametrize("bc_z", [0, 1])
def test_ghost_fill_of_a_single_shell(bc_z):
    """One cell in x: no ghosts there, and the y-z edges filled from the y and z faces
    (strips copied, means at the first and second diagonal), against plain numpy."""
    kc = koralcuda()
    kc.lib()
    src = kc.Sim(kc.puffy_grid(24, 9, 7), kc.puffy_options())
    src.initPuffy(1e-3, 1e-3, 5)
    grid, ng = kc.puffy_grid(1, 9, 7), 3
    assert grid.ng == ng
    sim = kc.Sim(grid, kc.puffy_options(bc_y=1, bc_z=bc_z))
    p = src.p.reshape(7 + 2 * ng, 9 + 2 * ng, 24 + 2 * ng, 13)[:, :, 15].copy()
    p[:, :, 2] = np.linspace(0.0, 1e-3, p[:, :, 2].size).reshape(p.shape[:2])  # no two cells alike
    sim.set_prims(p.reshape(-1, 13))
    sim.set_cons(np.full((p.shape[0] * p.shape[1], 13), np.nan))
    sim.setBc()

    def y(iy):
        return iy + ng

    z, want = y, p.copy()
    for i in range(1, ng + 1):  # faces
        want[ng:-ng, y(-i)], want[ng:-ng, y(8 + i)] = p[ng:-ng, y(0)], p[ng:-ng, y(8)]
        want[z(-i), ng:-ng] = p[z(7 - i if bc_z == 0 else 0), ng:-ng]
        want[z(6 + i), ng:-ng] = p[z(i - 1 if bc_z == 0 else 6), ng:-ng]
    face, filled = want.copy(), np.zeros(p.shape[:2], bool)
    for ys, ye in ((-1, 0), (1, 8)):
        for zs, ze in ((-1, 0), (1, 6)):
            for k in range(2, ng + 1):
                want[z(ze + zs), y(ye + k * ys)] = face[z(ze), y(ye + k * ys)]
                want[z(ze + k * zs), y(ye + ys)] = face[z(ze + k * zs), y(ye)]
            for k in (1, 2):
                want[z(ze + k * zs), y(ye + k * ys)] = 0.5 * (face[z(ze), y(ye + k * ys)] + face[z(ze + k * zs), y(ye)])
            for k in range(1, ng + 1):
                filled[z(ze + zs), y(ye + k * ys)] = filled[z(ze + k * zs), y(ye + ys)] = True
            filled[z(ze + 2 * zs), y(ye + 2 * ys)] = True
    assert np.array_equal(_bits(sim.p), _bits(want.reshape(-1, 13)))
    assert np.all(np.isfinite(sim.u.reshape(p.shape)[filled]))


@pytest.mark.parametrize("shape", [(45, 45, 1), (64, 32, 1), (50, 41, 1), (160, 129, 1), (61, 40, 12)])
def test_scalar_sums_around_the_fold_sizes(shape):
    """Up to 2048 terms folded by one warp, more in chunks of 1024: 2025, 2048,
    2050, 20640 and 29280 cells, shells inside the domain."""
    gpu, orc = _pair(*shape)
    a, b = gpu.scalars(0.1, 50.0, 15.0), orc.scalar_row(0.1, 50.0, 15.0)
    for k in a:
        assert np.float64(a[k]).view(np.uint64) == np.float64(b[k]).view(np.uint64), (k, a[k], b[k])


@pytest.mark.parametrize("n", [1, 31, 33, 1777, 7200])
def test_batch_forms_agree(n):
    """Batches of one cell, around a warp, and around and above the device's
    warps: the per-cell, persistent and sorted forms give the same bits."""
    kc = koralcuda()
    kc.lib()
    opt = kc.puffy_options()
    geom, dt, pp = kc.synth_implicit_cells(opt, n, 3)
    ref = kc.implicit_batch(opt, geom, dt, pp, mode=0)
    for mode in (1, 3, 5):
        got = kc.implicit_batch(opt, geom, dt, pp, mode=mode)
        assert np.array_equal(_bits(got[0]), _bits(ref[0])) and np.array_equal(got[1], ref[1])


@pytest.mark.parametrize("variant,opt", [
    (1, {"radimp_start_with_bisect": 0}), (2, {"radimp_scale_jacobian": 0}), (3, {"radimp_lag_opac": 1}),
    (4, {"radimp_allow_rad_ceiling": 0, "radimp_allow_entr_in_4dprim": 0}),
    (5, {"radimp_opdamp_maxlevels": 1, "radimp_maxiter": 9}), (12, {"radimp_opdamp_maxlevels": -1})])
def test_batch_options(lean_binary, cells, tmp_path, variant, opt):  # noqa: F811
    """The batch forms under the options that change the solve's path, lag_opac's
    own slots among them, against the plain solve on the host (lean_check.cpp's
    variants)."""
    path, n = cells
    out = tmp_path / "plain.bin"
    subprocess.run([lean_binary, path, str(n), str(variant), str(out)], check=True, capture_output=True)
    want = np.fromfile(out).reshape(n, 19)
    kc = koralcuda()
    kc.lib()
    a = np.fromfile(path).reshape(n, 37)
    for mode in (0, 1, 5):
        pp, res = kc.implicit_batch(kc.puffy_options(**opt), a[:, :23], a[:, 23], a[:, 24:], mode=mode)
        same = (_bits(pp) == _bits(want[:, :13])) | (np.isnan(pp) & np.isnan(want[:, :13]))
        assert same.all(), np.argwhere(~same)[:3]
        assert np.array_equal(res, want[:, 13:].astype(np.int32))


def _pairs(sim, cap=8192):
    x, t = sim.get_harvest(cap)
    return {r.tobytes() for r in np.concatenate([x, t], axis=1)}


def test_harvest_records_first_exits_under_the_guess():
    """With a guess installed, the cells whose pre-solve state already passes the
    first residual test are finished before the ladder; the unfiltered harvest
    records them all the same, as the run without a bisection does (its pairs less
    those of its filtered harvest)."""
    kc = koralcuda()
    kc.lib()
    grid = kc.puffy_grid(40, 30, 1)
    rng = np.random.default_rng(2)
    w = rng.normal(0.0, 0.05, kc.KC_MLP_NWEIGHTS)
    w[16:32], w[36:40] = 1.0, 1.0  # the standard deviations
    got = {}
    for guess in (False, True):
        for mode in (0, 1):
            sim = kc.Sim(grid, kc.puffy_options(radimp_start_with_bisect=0))
            sim.initPuffy(1e-3, 1e-3, 5)
            sim.step()
            dt = 1e-6 * sim.cflDt()  # short enough that some cells need no iteration
            if guess:
                sim.set_guess(w)
            sim.harvest_implicit(8192)
            sim.set_harvest_filter(mode)
            sim.debug_phase(5, dt)
            got[guess, mode] = _pairs(sim)
    first = got[False, 0] - got[False, 1]
    assert len(first) > 20 and first <= got[True, 0] and not first & got[True, 1]


@pytest.mark.parametrize("n", [1, 40000])
def test_batch_calls_refuse_null_arrays(n):
    """Each host array of the batch calls, below and above the size from which large
    arrays are copied by several threads."""
    kc = koralcuda()
    lib = kc.lib()
    opt = kc.puffy_options()
    arr = [np.zeros((n, 23)), np.zeros((n, 13)), np.zeros((n, 13)), np.zeros((n, 6), np.int32)]
    for k in range(4):
        p = [None if i == k else a.ctypes.data for i, a in enumerate(arr)]
        assert lib.kc_implicit_batch(ctypes.byref(opt), n, *p, 0) == kc.KC_ERR_INVALID_CONFIG
        assert lib.kc_u2p_batch(ctypes.byref(opt), n, *p) == kc.KC_ERR_INVALID_CONFIG


def _inversion_cells(kc, opt, n):
    """Seeded cells as inputs of the inversion: rows of primitives as conserveds are
    states like any other to it, solvable or not."""
    geom, _, pp = kc.synth_implicit_cells(opt, n, 11)
    uu = pp * geom[:, 20:21]
    uu[:, 1] = -uu[:, 0] - uu[:, 1]  # T^t_t
    uu[:, 9] = -uu[:, 9]
    return geom, uu, pp


def test_small_host_batches_alone_and_at_once():
    """Host-array calls whose arrays fit the fixed device array (5,188 cells of an
    inversion do, 5,190 do not), one after the other and from four threads, of which
    one at a time has it: the rows are those of one large call."""
    import threading

    kc = koralcuda()
    kc.lib()
    opt = kc.puffy_options()
    geom, uu, pp = _inversion_cells(kc, opt, 6000)
    ref = kc.u2p_batch(opt, geom, uu, pp)
    geo2, dt2, pp2 = kc.synth_implicit_cells(opt, 40, 4)
    ref2 = kc.implicit_batch(opt, geo2, dt2, pp2, mode=5)
    bad = []

    def calls(sizes):
        for n in sizes:
            got = kc.u2p_batch(opt, geom[:n], uu[:n], pp[:n])
            if not (np.array_equal(_bits(got[0]), _bits(ref[0][:n])) and np.array_equal(got[1], ref[1][:n])):
                bad.append(n)
        got = kc.implicit_batch(opt, geo2, dt2, pp2, mode=5)
        if not (np.array_equal(_bits(got[0]), _bits(ref2[0])) and np.array_equal(got[1], ref2[1])):
            bad.append("solve")

    calls([1, 5188, 5189, 5190, 33])
    th = [threading.Thread(target=calls, args=([n, 7 * n, 5188, n, 1] * 4,)) for n in (3, 100, 333, 740)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad
