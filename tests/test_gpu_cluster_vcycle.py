"""The lower levels of the V-cycle inside one cluster against the same levels as
one launch per step (PDEB200_NO_TAIL): two preconditioned CG iterations give
the same field. The two forms differ by roundings only (a reciprocal instead
of a division, exact zeros instead of residuals of the order of eps, the
coarsest sweeps as one matrix), about 100 roundings of 1e-16 per value and
V-cycle, amplified by two CG iterations: 1e-11 relative.

The grids put the first cluster level at the finest level or below it, with one
CTA or several per level, fewer layers than CTAs, coarsest levels of one
and of several nodes, semi-coarsened and non-nested levels."""
import numpy as np
import pytest

from pde_solver_b200 import abi, solver
from pde_solver_b200.problem import FaceBC, GridProblem, default_options

pytestmark = pytest.mark.gpu

MIXED = [FaceBC.dirichlet(0.1), FaceBC.neumann(0.1), FaceBC.robin(1.0, 1.0, 0.0), FaceBC.dirichlet(0.5),
         FaceBC.neumann(0.0), FaceBC.robin(2.0, 0.01, 0.1)]
DIRICHLET = [FaceBC.dirichlet(0.0)] * 6


@pytest.fixture(scope="module", autouse=True)
def _lib(lib):
    return lib


def rel_l2(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def make(dims, coef, faces, bounds=(0.0, 1.0, 0.0, 1.0, 0.0, 1.0)):
    rng = np.random.Generator(np.random.PCG64(sum(dims)))
    p = GridProblem(*dims, bounds=bounds, a=-1.0, b=-1.0, az=-1.0)
    if coef == "divk":
        p = GridProblem(*dims, bounds=bounds, coef_kind=abi.COEF_DIVK)
        p.k = np.exp(0.5 * rng.standard_normal(p.n))
    p.f = rng.standard_normal(p.n)
    p.faces = list(faces)
    return p


DIMS = [(5, 5, 1), (9, 9, 1), (33, 25, 1), (100, 37, 1), (129, 97, 1), (257, 130, 1), (7, 6, 5), (9, 9, 9),
        (17, 17, 17), (33, 33, 33), (34, 20, 27), (40, 9, 12), (12, 11, 70), (65, 65, 65), (66, 50, 44)]


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("coef", ["divk", "const"])
@pytest.mark.parametrize("faces", ["mixed", "dirichlet"])
@pytest.mark.parametrize("sweeps", [(2, 2), (1, 2), (3, 0)])
def test_cluster_levels_match_launches(monkeypatch, dims, coef, faces, sweeps):
    p = make(dims, coef, MIXED if faces == "mixed" else DIRICHLET)
    opt = default_options(method=abi.MG_PCG, tol=0.0, tol_mode=abi.TOL_RELATIVE, max_iter=2, mg_pre_smooth=sweeps[0],
                          mg_post_smooth=sweeps[1])
    a, ra = solver.solve(p, opt, raise_on_error=False)
    monkeypatch.setenv("PDEB200_NO_TAIL", "1")
    b, rb = solver.solve(p, opt, raise_on_error=False)
    assert ra.status == rb.status and ra.iterations == rb.iterations
    assert rel_l2(a, b) <= 1e-11


# What a CTA sends after the prolongation (nothing without sweeps after it) and
# in the sweeps that follow: one and two layers per CTA; every run gives the same bits.
@pytest.mark.parametrize("dims", [(17, 17, 18), (33, 33, 33), (40, 36, 20), (33, 40, 1), (129, 97, 1)])
@pytest.mark.parametrize("sweeps", [(2, 1), (1, 0), (1, 3)])
def test_cluster_levels_after_prolongation(monkeypatch, dims, sweeps):
    p = make(dims, "divk", MIXED)
    opt = default_options(method=abi.MG_PCG, tol=0.0, tol_mode=abi.TOL_RELATIVE, max_iter=2, mg_pre_smooth=sweeps[0],
                          mg_post_smooth=sweeps[1])
    a, _ = solver.solve(p, opt, raise_on_error=False)
    for _ in range(10):
        assert np.array_equal(solver.solve(p, opt, raise_on_error=False)[0], a)
    monkeypatch.setenv("PDEB200_NO_TAIL", "1")
    b, _ = solver.solve(p, opt, raise_on_error=False)
    assert rel_l2(a, b) <= 1e-11


def test_cluster_levels_semi_coarsened(monkeypatch):
    p = make((65, 33, 9), "divk", MIXED, bounds=(0.0, 4.0, 0.0, 1.0, 0.0, 0.1))
    opt = default_options(method=abi.MG_PCG, tol=0.0, tol_mode=abi.TOL_RELATIVE, max_iter=2)
    a, _ = solver.solve(p, opt, raise_on_error=False)
    monkeypatch.setenv("PDEB200_NO_TAIL", "1")
    b, _ = solver.solve(p, opt, raise_on_error=False)
    assert rel_l2(a, b) <= 1e-11


@pytest.mark.parametrize("bf16", [0, 1])
@pytest.mark.parametrize("dims", [(65, 49, 33), (200, 150, 1), (33, 33, 33)])
def test_cluster_levels_mixed_precision(oracle_mod, bf16, dims):
    p = make(dims, "divk", MIXED)
    opt = default_options(method=abi.MG_PCG, tol=1e-11, tol_mode=abi.TOL_RELATIVE, max_iter=200,
                          precision=abi.MIXED, bf16_coefficients=bf16)
    got, rep = solver.solve(p, opt)
    assert rep.status == abi.OK and rep.rel_residual <= 1e-11
    st, ref, _ = oracle_mod.rs_solve(p, default_options(method=abi.MG_PCG, tol=1e-13, tol_mode=abi.TOL_RELATIVE,
                                                        max_iter=300))
    assert st == 0 and rel_l2(got, ref) <= 1e-8  # the bar of the mixed form


def kernels_of(p, opt):
    """Names of the kernels that a solve launched under the profiler, without their level."""
    lib = abi.load()
    lib.pdeb200_profile_enable(0, 1)
    try:
        solver.solve(p, opt, raise_on_error=False)
        stats = (abi.KernelStat * 256)()
        n = lib.pdeb200_profile_read(0, stats, 256)
    finally:
        lib.pdeb200_profile_enable(0, 0)
    return {stats[q].name.decode().split("@")[0] for q in range(n)}


# Robin faces with a value per node: the transfer tables do not hold them, and the
# levels below about 1100 nodes run in one block as they did before there was a
# cluster form. Levels through the cluster else.
@pytest.mark.parametrize("dims", [(33, 33, 33), (100, 37, 1), (34, 20, 27), (65, 40, 5)])
def test_levels_with_closures_per_node(monkeypatch, dims):
    p = make(dims, "const", MIXED)
    opt = default_options(method=abi.MG_PCG, tol=0.0, tol_mode=abi.TOL_RELATIVE, max_iter=2)
    used = kernels_of(p, opt)
    assert "cluster_vcycle" in used and "tail_vcycle" not in used
    nx, ny, nz = dims
    rng = np.random.Generator(np.random.PCG64(nx))
    p.faces[2] = FaceBC(abi.BC_ROBIN, alpha=1.0, beta=0.5, gamma=0.1, alpha_arr=1.0 + rng.random(nx * nz))
    p.faces[0] = FaceBC(abi.BC_ROBIN, alpha=1.0, beta=0.5, gamma=0.1, beta_arr=0.1 + rng.random(ny * nz))
    used = kernels_of(p, opt)
    assert "tail_vcycle" in used and "cluster_vcycle" not in used
    a, ra = solver.solve(p, opt, raise_on_error=False)
    monkeypatch.setenv("PDEB200_NO_TAIL", "1")
    b, rb = solver.solve(p, opt, raise_on_error=False)
    assert ra.iterations == rb.iterations and rel_l2(a, b) <= 1e-11


# More than 65536 planes: a fine plane's number times the coarse intervals does not
# fit in 32 bits. Nested and not nested, coarsened along z only; as many
# iterations as on a grid where it does.
@pytest.mark.parametrize("nz", [70000, 70001])
def test_prolongation_of_many_planes(nz):
    its = []
    for planes in (nz, nz - 10000):
        p = GridProblem(3, 3, planes, bounds=(0.0, 1.0, 0.0, 1.0, 0.0, planes / 2.0), a=-1.0, b=-1.0, az=-1.0, e=0.05)
        p.f = np.random.Generator(np.random.PCG64(7)).standard_normal(p.n)
        p.faces = [FaceBC.neumann(0.0)] * 4 + [FaceBC.dirichlet(0.0)] * 2
        got, rep = solver.solve(p, default_options(method=abi.MG_PCG, tol=1e-10, tol_mode=abi.TOL_RELATIVE, max_iter=60))
        assert rep.status == abi.OK and rep.rel_residual <= 1.1e-10
        its.append(rep.iterations)
    assert abs(its[0] - its[1]) <= 1 and its[0] <= 30
