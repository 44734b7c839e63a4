"""The launch forms of the MG-PCG solve change no numbers: replaying each PCG
iteration as a captured CUDA graph or launching kernel by kernel, and
launching with programmatic stream serialization (each kernel may be
scheduled while its predecessor drains, and waits for it before touching
memory) or in plain stream order, give bit-identical fields and the same
iteration count."""
import os
import subprocess
import sys

import numpy as np
import pytest

from pde_solver_b200 import abi, solver, synthetic
from pde_solver_b200.problem import FaceBC, GridProblem, default_options

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _problem(n=65):
    p = synthetic.varcoef_poisson_3d(n, seed=5)
    p.faces = [FaceBC.dirichlet(0.0), FaceBC.neumann(0.1), FaceBC.robin(1.0, 1.0, 0.0), FaceBC.dirichlet(0.5),
               FaceBC.neumann(0.0), FaceBC.robin(2.0, 0.5, 0.1)]
    return p


def _opt():
    return default_options(method=abi.MG_PCG, tol=1e-10, tol_mode=abi.TOL_RELATIVE, max_iter=200)


@pytest.fixture(scope="module", autouse=True)
def _lib(lib):
    return lib


def test_graph_replay_changes_no_numbers(monkeypatch):
    p = _problem()
    a, ra = solver.solve(p, _opt())
    monkeypatch.setenv("PDEB200_NO_GRAPH", "1")
    b, rb = solver.solve(p, _opt())
    assert ra.iterations == rb.iterations and ra.iterations > 0
    assert np.array_equal(a, b)


def test_programmatic_launch_changes_no_numbers(tmp_path):
    # the launch attribute is chosen once per device context, so the plain
    # stream-order solve runs in a child process
    p = _problem()
    a, ra = solver.solve(p, _opt())
    out = tmp_path / "plain.npy"
    code = (
        "import sys, numpy as np\n"
        f"sys.path.insert(0, {REPO!r})\n"
        f"sys.path.insert(0, {os.path.join(REPO, 'tests')!r})\n"
        "from test_gpu_launch_forms import _problem, _opt\n"
        "from pde_solver_b200 import solver\n"
        "u, r = solver.solve(_problem(), _opt())\n"
        f"np.save({str(out)!r}, u)\n"
        "print(r.iterations)\n"
    )
    env = dict(os.environ, PDEB200_NO_PDL="1")
    res = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
    assert res.returncode == 0, res.stderr[-2000:]
    assert int(res.stdout.strip().splitlines()[-1]) == ra.iterations
    assert np.array_equal(np.load(out), a)


# Several inner solves per refinement, each of three and more iterations: every
# one starts from its own residual, whether its iterations are replayed or not.
# Levels by launches, so that an iteration has enough of them to be captured.
@pytest.mark.parametrize("dims", [(49, 49, 49), (41, 53, 37), (150, 140, 1)])
def test_graph_replay_changes_no_numbers_in_refinement(monkeypatch, dims):
    nx, ny, nz = dims
    p = GridProblem(nx, ny, nz, a=-1.0, b=-1.0, az=-1.0, c=30.0, d=-20.0, dz=10.0 if nz > 1 else 0.0)
    p.f = np.random.Generator(np.random.PCG64(nx)).standard_normal(p.n)
    opt = default_options(method=abi.MG_BICGSTAB, precision=abi.MIXED, tol=1e-12, tol_mode=abi.TOL_RELATIVE,
                          max_iter=400)
    monkeypatch.setenv("PDEB200_NO_TAIL", "1")
    a, ra = solver.solve(p, opt)
    monkeypatch.setenv("PDEB200_NO_GRAPH", "1")
    b, rb = solver.solve(p, opt)
    assert ra.status == abi.OK and ra.iterations == rb.iterations and ra.iterations >= 6
    assert np.array_equal(a, b)


def test_graph_replay_of_a_long_solve_of_few_launches(monkeypatch):
    # two levels and closures per node: no cluster kernel, at most 24 launches per
    # iteration, captured late
    p = GridProblem(48, 54, 13, a=-1.0, b=-1.0, az=-1.0)
    rng = np.random.Generator(np.random.PCG64(2))
    p.f = rng.standard_normal(p.n)
    p.faces[0] = FaceBC(abi.BC_ROBIN, alpha=1.5, beta=0.1, gamma=0.2, alpha_arr=1.0 + rng.random(54 * 13))
    opt = default_options(method=abi.MG_PCG, tol=0.0, tol_mode=abi.TOL_RELATIVE, max_iter=45, mg_max_levels=2,
                          mg_coarse_iters=1)
    a, ra = solver.solve(p, opt, raise_on_error=False)
    monkeypatch.setenv("PDEB200_NO_GRAPH", "1")
    b, rb = solver.solve(p, opt, raise_on_error=False)
    assert ra.iterations == rb.iterations == 45 and np.array_equal(a, b)
