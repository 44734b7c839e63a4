"""The red-black sweep in one pass (PDEB200_PAIR_MIN lowered) against two colour
passes: two preconditioned CG iterations give the same field. The node updates
are the same arithmetic (the r.z sum has another order), so about 100 roundings
of 1e-16 per value and V-cycle, amplified by two CG iterations: 1e-11 relative.

The grids put the tile (30 columns by 22 rows, 30 in FP32) and chunk (16 planes)
edges inside, at and next to the grid's; sweeps 1 to 3 before and after, odd
counts ending in the other buffer."""
import numpy as np
import pytest

from pde_solver_b200 import abi, solver
from pde_solver_b200.problem import FaceBC, GridProblem, default_options

pytestmark = pytest.mark.gpu

MIXED = [FaceBC.dirichlet(0.1), FaceBC.neumann(0.1), FaceBC.robin(1.0, 1.0, 0.0), FaceBC.dirichlet(0.5),
         FaceBC.neumann(0.0), FaceBC.robin(2.0, 0.01, 0.1)]
DIMS = [(20, 17, 12), (32, 24, 18), (33, 25, 35), (62, 32, 20), (61, 47, 51), (5, 90, 40)]


@pytest.fixture(scope="module", autouse=True)
def _lib(lib):
    return lib


def make(dims, sparse=False):
    rng = np.random.Generator(np.random.PCG64(sum(dims)))
    p = GridProblem(*dims, a=-1.0, b=-1.0, az=-1.0)
    p.f = rng.standard_normal(p.n)
    if sparse:  # mostly zero right-hand side: the updates' zero dividends
        p.f[rng.random(p.n) < 0.99] = 0.0
    p.faces = [FaceBC.dirichlet(0.0)] * 6 if sparse else list(MIXED)
    return p


def both(monkeypatch, p, opt):
    monkeypatch.setenv("PDEB200_NO_TAIL", "1")
    monkeypatch.setenv("PDEB200_PAIR_MIN", "1000")
    a, ra = solver.solve(p, opt, raise_on_error=False)
    monkeypatch.setenv("PDEB200_PAIR_MIN", str(1 << 40))
    b, rb = solver.solve(p, opt, raise_on_error=False)
    assert ra.status == rb.status
    return a, b, ra, rb


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("sweeps", [(2, 2), (1, 2), (3, 1), (2, 3), (0, 1)])
@pytest.mark.parametrize("sparse", [False, True])
def test_one_pass_matches_colour_passes(monkeypatch, dims, sweeps, sparse):
    opt = default_options(method=abi.MG_PCG, tol=0.0, tol_mode=abi.TOL_RELATIVE, max_iter=2, mg_pre_smooth=sweeps[0],
                          mg_post_smooth=sweeps[1])
    a, b, ra, rb = both(monkeypatch, make(dims, sparse), opt)
    assert ra.iterations == rb.iterations
    assert np.linalg.norm(a - b) <= 1e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("dims", DIMS[:5])
def test_one_pass_in_mixed_precision(monkeypatch, dims):
    # FP32 sweeps: both forms converge, in as many inner iterations give or take
    # one, to fields that differ by the mixed form's bar
    opt = default_options(method=abi.MG_PCG, tol=1e-11, tol_mode=abi.TOL_RELATIVE, max_iter=200, precision=abi.MIXED)
    a, b, ra, rb = both(monkeypatch, make(dims), opt)
    assert ra.status == abi.OK and ra.rel_residual <= 1e-11
    assert abs(ra.iterations - rb.iterations) <= 1
    assert np.linalg.norm(a - b) <= 1e-8 * np.linalg.norm(b)


@pytest.mark.parametrize("dims", DIMS[:5])
@pytest.mark.parametrize("sweeps", [(2, 2), (1, 1)])
def test_bicgstab_on_column_kernels(monkeypatch, dims, sweeps):
    # MG-BiCGStab with the apply and its sums in one launch (k_apply_columns,
    # 32 x 16 columns) against separate ones, in both output buffers of the
    # V-cycle: two iterations, whose scalars amplify the roundings of differently
    # ordered sums by up to 1e5: 1e-9 relative
    p = make(dims)
    p.c, p.d, p.dz = 3.0, -2.0, 1.0
    opt = default_options(method=abi.MG_BICGSTAB, tol=0.0, tol_mode=abi.TOL_RELATIVE, max_iter=2,
                          mg_pre_smooth=sweeps[0], mg_post_smooth=sweeps[1])
    a, b, ra, rb = both(monkeypatch, p, opt)
    assert ra.iterations == rb.iterations
    assert np.linalg.norm(a - b) <= 1e-9 * np.linalg.norm(b)


@pytest.mark.parametrize("dims", DIMS[:5])
def test_bicgstab_in_mixed_precision_on_column_kernels(monkeypatch, dims):
    p = make(dims)
    p.c, p.d, p.dz = 3.0, -2.0, 1.0
    opt = default_options(method=abi.MG_BICGSTAB, tol=1e-10, tol_mode=abi.TOL_RELATIVE, max_iter=200,
                          precision=abi.MIXED)
    a, b, ra, rb = both(monkeypatch, p, opt)
    assert ra.status == abi.OK and ra.rel_residual <= 1e-10
    assert np.linalg.norm(a - b) <= 1e-8 * np.linalg.norm(b)  # the bar of the mixed form


def make_divk(dims):
    p = make(dims)
    q = GridProblem(*dims, coef_kind=abi.COEF_DIVK)
    q.k = np.exp(0.5 * np.random.Generator(np.random.PCG64(7)).standard_normal(q.n))
    q.f, q.faces = p.f, p.faces
    return q


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("sweeps", [(2, 2), (1, 2), (3, 1)])
def test_one_pass_with_sampled_k(monkeypatch, dims, sweeps):
    opt = default_options(method=abi.MG_PCG, tol=0.0, tol_mode=abi.TOL_RELATIVE, max_iter=2, mg_pre_smooth=sweeps[0],
                          mg_post_smooth=sweeps[1])
    a, b, ra, rb = both(monkeypatch, make_divk(dims), opt)
    assert ra.iterations == rb.iterations
    assert np.linalg.norm(a - b) <= 1e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("dims", DIMS[:5])
@pytest.mark.parametrize("bf16", [0, 1])
def test_one_pass_with_sampled_k_in_mixed_precision(monkeypatch, dims, bf16):
    opt = default_options(method=abi.MG_PCG, tol=1e-11, tol_mode=abi.TOL_RELATIVE, max_iter=200, precision=abi.MIXED,
                          bf16_coefficients=bf16)
    a, b, ra, rb = both(monkeypatch, make_divk(dims), opt)
    assert ra.status == abi.OK and ra.rel_residual <= 1e-11
    assert abs(ra.iterations - rb.iterations) <= 1
    assert np.linalg.norm(a - b) <= 1e-8 * np.linalg.norm(b)
