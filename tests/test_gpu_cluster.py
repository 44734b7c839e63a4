"""Relaxation runs and heat steps held in the shared memory of one thread-block
cluster (Jacobi, lexicographic Gauss-Seidel / SOR, forward Euler) against the oracle, at the sizes
where the slabs, the sweep batches and the launches change: one layer per CTA
and fewer layers than CTAs, rows of odd and even length, sweep counts around the
batch and launch sizes, stopping inside a batch.

Tolerance: a sweep is a contraction of the error, and each adds a few
roundings (FMA contraction is the only difference), so after S sweeps the
fields differ by at most about 10 S eps relative: 1e-11 for S <= 4500."""
import ctypes

import numpy as np
import pytest

from pde_solver_b200 import abi, solver
from pde_solver_b200.problem import FaceBC, GridProblem, default_options

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(lib):
    return lib


def rel_l2(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def make(dims, coef="const", faces="mixed", seed=3):
    rng = np.random.Generator(np.random.PCG64(seed))
    p = GridProblem(*dims, a=-1.0, b=-0.8, az=-1.2, c=0.3, e=-0.2)
    nx, ny, nz = dims
    if coef == "divk":
        p = GridProblem(*dims, coef_kind=abi.COEF_DIVK)
        p.k = np.exp(0.3 * rng.standard_normal(p.n))
    elif coef == "nodal":
        p = GridProblem(*dims, coef_kind=abi.COEF_NODAL)
        o = np.ones(p.n)
        p.nodal = np.concatenate([-o - rng.random(p.n), -o, -o, 0.2 * o, 0 * o, 0 * o, 0 * o])
    if faces == "mixed":
        p.faces = [FaceBC.robin(1.0, 0.5, 0.2), FaceBC.dirichlet(0.3), FaceBC.neumann(0.3), FaceBC.dirichlet(1.0),
                   FaceBC.neumann(-0.2), FaceBC.robin(2.0, 0.01, 0.1)]
    elif faces == "arrays":
        p.faces = [FaceBC(abi.BC_NEUMANN, value_arr=rng.standard_normal(ny * nz)),
                   FaceBC(abi.BC_DIRICHLET, value_arr=rng.standard_normal(ny * nz)),
                   FaceBC(abi.BC_DIRICHLET, value_arr=rng.standard_normal(nx * nz)),
                   FaceBC(abi.BC_ROBIN, alpha=2.0, beta=0.01, gamma_arr=rng.standard_normal(nx * nz)),
                   FaceBC(abi.BC_DIRICHLET, value_arr=rng.standard_normal(nx * ny)), FaceBC.neumann(0.1)]
    p.f = rng.standard_normal(p.n)
    return p


def check(oracle_mod, p, bar=1e-11, **kw):
    opt = default_options(**kw)
    got, rep = solver.solve(p, opt)
    st, ref, rrep = oracle_mod.rs_solve(p, opt)
    # the reference returns its field without an error at the sweep limit
    assert st == 0 and rep.status == (abi.OK if rep.last_delta < opt.tol else abi.ERR_NOT_CONVERGED)
    assert rep.iterations == rrep.iterations
    assert rel_l2(got, ref) <= bar
    if rrep.last_delta > 0:
        assert abs(rep.last_delta - rrep.last_delta) <= 1e-6 * rrep.last_delta + 1e-13


@pytest.mark.parametrize("method", [abi.JACOBI, abi.GAUSS_SEIDEL, abi.SOR])
@pytest.mark.parametrize("dims", [(3, 3, 1), (3, 40, 1), (40, 3, 1), (36, 35, 1), (97, 65, 1), (130, 67, 1),
                                  (3, 3, 3), (12, 11, 5), (20, 19, 35)])
@pytest.mark.parametrize("faces", ["mixed", "arrays"])
def test_cluster_relaxation_sizes(oracle_mod, method, dims, faces):
    check(oracle_mod, make(dims, faces=faces), method=method, max_iter=40, tol=0.0)


@pytest.mark.parametrize("method", [abi.JACOBI, abi.SOR])
@pytest.mark.parametrize("sweeps", [1, 2, 64, 65, 66, 193, 194, 1000, 2047, 2048, 2049, 4100])
def test_cluster_relaxation_sweep_counts(oracle_mod, method, sweeps):
    check(oracle_mod, make((23, 18, 1)), method=method, max_iter=sweeps, tol=0.0)


# The last maximum is the one of the field's own nodes, to the bit: the fields of
# S and S - 1 sweeps give it. Slabs whose threads have one node fewer than
# others, on several CTAs.
@pytest.mark.parametrize("dims", [(36, 35, 1), (97, 65, 1), (131, 67, 1), (129, 129, 1), (20, 19, 35)])
@pytest.mark.parametrize("sweeps", [2, 41, 150])
def test_cluster_jacobi_last_delta_is_of_the_field(dims, sweeps):
    p = make(dims)
    a, ra = solver.solve(p, default_options(method=abi.JACOBI, max_iter=sweeps, tol=0.0))
    b, rb = solver.solve(p, default_options(method=abi.JACOBI, max_iter=sweeps - 1, tol=0.0))
    inner = (slice(1, -1),) * (3 if dims[2] > 1 else 2)
    shape = (dims[2], dims[1], dims[0]) if dims[2] > 1 else (dims[1], dims[0])
    assert ra.iterations == sweeps and rb.iterations == sweeps - 1
    assert ra.last_delta == np.abs(a - b).reshape(shape)[inner].max()


# Runs of few sweeps in one block, of more in a cluster (from 4 sweeps on, 7 or 8
# on the larger grids).
@pytest.mark.parametrize("dims", [(23, 18, 1), (97, 65, 1), (200, 180, 1), (20, 19, 35), (1200, 3, 1)])
@pytest.mark.parametrize("sweeps", [3, 4, 5, 6, 7, 8, 9])
def test_lexicographic_few_sweeps(oracle_mod, dims, sweeps):
    check(oracle_mod, make(dims), method=abi.GAUSS_SEIDEL, max_iter=sweeps, tol=0.0)


# A batch shorter than the one before it (the last before the sweep limit: 64,
# 128 .. 512 sweeps, then 1 or 2): every warp takes the same branch after each
# batch. One launch form only, so each run gives the same bits; against the
# oracle once.
@pytest.mark.parametrize("dims", [(36, 35, 1), (97, 65, 1), (20, 19, 35)])
@pytest.mark.parametrize("sweeps", [66, 67, 194, 450, 963])
def test_cluster_lexicographic_short_last_batch(oracle_mod, dims, sweeps):
    p = make(dims)
    opt = default_options(method=abi.SOR, max_iter=sweeps, tol=0.0)
    check(oracle_mod, p, method=abi.SOR, max_iter=sweeps, tol=0.0)
    first, r0 = solver.solve(p, opt)
    for _ in range(10):
        got, rep = solver.solve(p, opt)
        assert (rep.iterations, rep.last_delta) == (r0.iterations, r0.last_delta)
        assert np.array_equal(got, first)


# Stopping inside a batch with one plane per CTA and an odd last hyperplane: the
# sweeps that are run again and the last one send the same nodes in a row.
@pytest.mark.parametrize("dims", [(21, 18, 18), (18, 21, 18), (22, 18, 18)])
@pytest.mark.parametrize("tol", [1e-2, 1e-4, 1e-6])
def test_cluster_lexicographic_rerun_then_last_sweep(oracle_mod, dims, tol):
    p = make(dims)
    opt = default_options(method=abi.SOR, max_iter=20000, tol=tol)
    check(oracle_mod, p, method=abi.SOR, max_iter=20000, tol=tol)
    first, r0 = solver.solve(p, opt)
    for _ in range(10):
        got, rep = solver.solve(p, opt)
        assert (rep.iterations, rep.last_delta) == (r0.iterations, r0.last_delta)
        assert np.array_equal(got, first)


@pytest.mark.parametrize("method", [abi.JACOBI, abi.SOR])
@pytest.mark.parametrize("tol", [1.0, 1e-2, 1e-3, 1e-5, 1e-7])
@pytest.mark.parametrize("dims", [(31, 44, 1), (13, 14, 15)])
def test_cluster_relaxation_stops_where_the_oracle_stops(oracle_mod, method, dims, tol):
    check(oracle_mod, make(dims), method=method, max_iter=20000, tol=tol)


@pytest.mark.parametrize("method", [abi.JACOBI, abi.GAUSS_SEIDEL])
@pytest.mark.parametrize("coef", ["divk", "nodal"])
@pytest.mark.parametrize("dims", [(45, 38, 1), (14, 13, 12)])
def test_cluster_relaxation_coefficients(oracle_mod, method, coef, dims):
    check(oracle_mod, make(dims, coef), method=method, max_iter=150, tol=0.0)


@pytest.mark.parametrize("method", [abi.JACOBI, abi.SOR])
def test_cluster_relaxation_constant_f_and_nonlinear(oracle_mod, method):
    p = make((37, 22, 1))
    p.f = None
    p.f_const = 0.7
    check(oracle_mod, p, method=method, max_iter=90, tol=0.0)
    p.nonlinear = [(abi.NL_POWER, 0.4, 2), (abi.NL_SIN, -0.3, 1)]
    check(oracle_mod, p, method=method, max_iter=90, tol=0.0)


# the last grid is too large for a cluster: one launch per step
@pytest.mark.parametrize("dims", [(3, 3, 1), (70, 41, 1), (9, 130, 1), (3, 4, 5), (19, 18, 20), (400, 401, 1)])
@pytest.mark.parametrize("faces", ["mixed", "arrays"])
def test_time_series_frames_and_boundaries(oracle_mod, dims, faces):
    p = make(dims, faces=faces)
    p.ut = 1.0
    p.u0 = np.random.Generator(np.random.PCG64(1)).standard_normal(p.n)
    h = min(1.0 / (d - 1) for d in dims if d > 1)
    dt = 0.2 * h * h / 2.4
    seen = {}
    got, rep = solver.time_series(p, 0.0, dt, 24, on_frame=lambda q, t, u: seen.__setitem__(q, u), frame_stride=7)
    ref, frames = oracle_mod.rs_time_series(p, 0.0, dt, 24, keep_frames=True)
    assert rep.iterations == 23 and sorted(seen) == [0, 7, 14, 21, 23]
    assert rel_l2(got, ref) <= 1e-12
    for q, u in seen.items():
        assert rel_l2(u, frames[q]) <= 1e-12
    assert np.array_equal(got, seen[23])


# The steps between two frames run one per launch or all in one, by their number
# and the grid's size: the same bits.
@pytest.mark.parametrize("dims", [(3, 3, 1), (70, 41, 1), (300, 200, 1), (3, 4, 5), (19, 18, 20)])
@pytest.mark.parametrize("coef", ["const", "divk"])
def test_time_series_frame_stride_changes_no_bit(dims, coef):
    p = make(dims, coef)
    p.ut = 1.0
    p.u0 = np.random.Generator(np.random.PCG64(1)).standard_normal(p.n)
    dt = 0.05 * min(1.0 / (d - 1) for d in dims if d > 1) ** 2
    frames = {}
    for stride in (1, 2, 3, 4, 8, 100):
        seen = {}
        got, rep = solver.time_series(p, 0.0, dt, 26, on_frame=lambda q, t, u: seen.__setitem__(q, u),
                                      frame_stride=stride)
        assert rep.iterations == 25 and sorted(seen) == sorted(set(range(0, 26, stride)) | {25})
        frames = frames or seen
        assert np.array_equal(got, frames[25])
        for q, u in seen.items():
            assert np.array_equal(u, frames[q])


# Krylov loops: the grids are held in shared memory, then with x, r and q in
# global memory, then by a launch per step. Both sides stop at the same
# tolerance, so the fields agree to that tolerance times the operator's
# condition (at most 1e5 here): the 1e-9 bar of the reference CG at tol 1e-12 |b|.
@pytest.mark.parametrize("dims", [(3, 3, 1), (5, 40, 1), (40, 5, 1), (130, 77, 1), (20, 19, 18), (300, 290, 1),
                                  (690, 650, 1)])
@pytest.mark.parametrize("relative", [False, True])
def test_cluster_cg_sizes(oracle_mod, dims, relative):
    p = GridProblem(*dims, a=-1.0, b=-2.0, az=-1.0, e=-0.5)
    x, y, z = p.coords()
    p.f = np.broadcast_to(np.sin(3.0 * x) * np.cos(2.0 * y) + 0.5 * z, (max(dims[2], 1), dims[1], dims[0])).reshape(-1).copy()
    bn = np.linalg.norm(p.f)
    opt = default_options(method=abi.CG, max_iter=6000, tol=1e-12 * (1.0 if relative else bn),
                          tol_mode=abi.TOL_RELATIVE if relative else abi.TOL_REFERENCE)
    got, rep = solver.solve(p, opt)
    st, ref, rrep = oracle_mod.rs_solve(p, default_options(method=abi.CG, max_iter=6000, tol=1e-12 * bn))
    assert st == 0 and rep.status == abi.OK
    assert abs(rep.iterations - rrep.iterations) <= 2 + rrep.iterations // 50
    assert rel_l2(got, ref) <= 1e-9


@pytest.mark.parametrize("sweeps", [1, 7])
def test_cluster_cg_iteration_limit(oracle_mod, sweeps):
    p = make((41, 38, 1), faces="none")
    opt = default_options(method=abi.CG, max_iter=sweeps, tol=1e-14)
    got, rep = solver.solve(p, opt)
    assert rep.status == abi.ERR_NOT_CONVERGED and rep.iterations == sweeps
    st, ref, rrep = oracle_mod.rs_solve(p, opt)
    assert rrep.iterations == sweeps and rel_l2(got, ref) <= 1e-11


@pytest.mark.parametrize("dims", [(4, 3, 1), (33, 60, 1), (17, 16, 15), (300, 280, 1), (60, 50, 40)])
def test_cluster_projection_sizes(oracle_mod, dims):
    nx, ny, nz = dims
    rng = np.random.Generator(np.random.PCG64(nx))
    n = nx * ny * nz
    u, v = rng.standard_normal(n), rng.standard_normal(n)
    w = rng.standard_normal(n) if nz > 1 else None
    h = 1.0 / 40
    a = (u, v, w, np.zeros(n), nx, ny, nz, h, h, h, 0.01, 20000, 1e-11)
    ug, vg, wg, pg, rep = solver.project_velocity(*a)
    _, ur, vr, wr, pr, rrep = oracle_mod.rs_project(*a)
    assert rep.success == rrep.success
    assert abs(rep.poisson_iterations - rrep.poisson_iterations) <= 2 + rrep.poisson_iterations // 50
    for g, r in ((ug, ur), (vg, vr), (pg, pr)) + (((wg, wr),) if nz > 1 else ()):
        assert rel_l2(g, r) <= 1e-8


# A negative limit makes no iteration.
@pytest.mark.parametrize("max_iter", [-3, -1])
@pytest.mark.parametrize("dims", [(33, 60, 1), (17, 16, 15)])
def test_cluster_projection_iteration_limit(oracle_mod, dims, max_iter):
    nx, ny, nz = dims
    rng = np.random.Generator(np.random.PCG64(ny))
    u, v, w, p = rng.standard_normal((4, nx * ny * nz))
    a = (u, v, w if nz > 1 else None, p, nx, ny, nz, 0.02, 0.03, 0.025, 0.01, max_iter, 1e-30)
    ug, vg, _, pg, rep = solver.project_velocity(*a)
    _, ur, vr, _, pr, rrep = oracle_mod.rs_project(*a)
    assert (rep.success, rep.poisson_iterations) == (rrep.success, rrep.poisson_iterations)
    assert rel_l2(ug, ur) <= 1e-12 and rel_l2(vg, vr) <= 1e-12 and rel_l2(pg, pr) <= 1e-12


# One and several virtual blocks and rounds; the 3D grid is served by launches. Both sides stop at a true residual of 1e-9 |b|, so the fields differ by
# at most 2e-9 times the condition number, about (n / 2)^2 in n nodes a side.
@pytest.mark.parametrize("dims", [(3, 3, 1), (3, 50, 1), (6, 40, 1), (40, 6, 1), (97, 81, 1), (161, 150, 1),
                                  (20, 19, 18)])
@pytest.mark.parametrize("coef", ["const", "nodal"])
@pytest.mark.parametrize("relative", [False, True])
def test_cluster_bicgstab_sizes(oracle_mod, dims, coef, relative):
    p = make(dims, coef, faces="none")
    x, y, z = p.coords()
    p.f = np.broadcast_to(np.sin(3.0 * x) * np.cos(2.0 * y) + 0.5 * z, (max(dims[2], 1), dims[1], dims[0])).reshape(-1).copy()
    bn = np.linalg.norm(p.f)
    opt = default_options(method=abi.BICGSTAB, max_iter=6000, tol=1e-9 * (1.0 if relative else bn),
                          tol_mode=abi.TOL_RELATIVE if relative else abi.TOL_REFERENCE)
    got, rep = solver.solve(p, opt)
    st, ref, _ = oracle_mod.rs_solve(p, default_options(method=abi.BICGSTAB, max_iter=6000, tol=1e-9 * bn))
    assert st == 0 and rep.status == abi.OK and rep.residual_l2 <= 1.01e-9 * bn
    assert rel_l2(got, ref) <= 2e-9 * (max(dims) / 2) ** 2


@pytest.mark.parametrize("iterations", [1, 2, 9])
def test_cluster_bicgstab_iteration_limit(oracle_mod, iterations):
    p = make((41, 38, 1), "nodal", faces="none")
    opt = default_options(method=abi.BICGSTAB, max_iter=iterations, tol=1e-14)
    got, rep = solver.solve(p, opt)
    st, ref, rrep = oracle_mod.rs_solve(p, opt)
    assert rep.status == abi.ERR_NOT_CONVERGED and rep.iterations == rrep.iterations == iterations
    assert rel_l2(got, ref) <= 1e-9


# A cancel flag is seen after the first sweeps (8) or iteration, on grids held by
# a cluster and by launches; a flag that stays 0 changes no bit.
@pytest.mark.parametrize("method, first", [(abi.JACOBI, 8), (abi.CG, 1), (abi.BICGSTAB, 1)])
@pytest.mark.parametrize("dims", [(41, 38, 1), (700, 690, 1)])
def test_cancel_is_seen_between_iterations(method, first, dims):
    p = make(dims, faces="none")
    p.c = 0.0
    opt = default_options(method=method, max_iter=150, tol=1e-13)
    ref, rref = solver.solve(p, opt, raise_on_error=False)
    flag = ctypes.c_int32(0)
    opt.cancel = ctypes.pointer(flag)
    got, rep = solver.solve(p, opt, raise_on_error=False)
    assert (rep.status, rep.iterations) == (rref.status, rref.iterations) and np.array_equal(got, ref)
    flag.value = 1
    _, rep = solver.solve(p, opt, raise_on_error=False)
    assert rep.status == abi.ERR_CANCELLED and rep.iterations == first
