"""Relaxation runs held in the shared memory of one thread-block cluster
(Jacobi, lexicographic Gauss-Seidel / SOR) against the oracle, at the sizes
where the slabs, the sweep batches and the launches change: one layer per CTA
and fewer layers than CTAs, rows of odd and even length, sweep counts around the
batch and launch sizes, stopping inside a batch.

Tolerance: a sweep is a contraction of the error, and each adds a few
roundings (FMA contraction is the only difference), so after S sweeps the
fields differ by at most about 10 S eps relative: 1e-11 for S <= 4500."""
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
