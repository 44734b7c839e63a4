"""The cluster kernels' quotients by one divisor (RoundedDiv) are those of the
correctly rounded division, to the bit: a Jacobi sweep of the zero field without
neighbour weights is -f / e, and heat steps without an operator add -f / u_t
each. Dividends over all exponents with random significands, subnormal, zero,
infinite, NaN; divisors inside and outside the range that the short form takes,
at its ends, with all bits of the significand set and one."""
import numpy as np
import pytest

from pde_solver_b200 import abi, solver
from pde_solver_b200.problem import GridProblem, default_options

pytestmark = pytest.mark.gpu

NX, NY = 131, 98
ONES = np.nextafter(2.0, 0.0)  # all bits of the significand set
EDGES = [1.0, 3.0, ONES, ONES * 2.0**-30, 1.0 + 2.0**-52, 2.0**-39, 2.0**199, np.nextafter(2.0**200, 0.0), 2.0**200,
         2.0**201, ONES * 2.0**300, 1e300, 1.7e308, 49152.0, 1e-11]


@pytest.fixture(scope="module", autouse=True)
def _lib(lib):
    return lib


def dividends(seed, lo=-1074, hi=1023):
    rng = np.random.Generator(np.random.PCG64(seed))
    m = 1.0 + rng.random((NY, NX))
    m[rng.random((NY, NX)) < 0.1] = ONES
    m[rng.random((NY, NX)) < 0.1] = 1.0
    f = np.ldexp(m, rng.integers(lo, hi + 1, (NY, NX))) * rng.choice([-1.0, 1.0], (NY, NX))
    special = [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, np.finfo(float).max, 2.0**-600, np.nextafter(2.0**-600, 0.0),
               2.0**600, np.nextafter(2.0**600, 0.0), np.finfo(float).tiny]
    f[1, 1:1 + len(special)] = special
    return f


def divisors(seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    return EDGES + list(np.ldexp(1.0 + rng.random(25), rng.integers(-30, 220, 25)))


def same(a, b):
    return np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("seed, lo, hi", [(1, -1074, 1023), (2, -650, 650), (3, -20, 20)])
def test_jacobi_quotients(seed, lo, hi):
    f = dividends(seed, lo, hi)
    for e in divisors(seed):
        p = GridProblem(NX, NY, 1, e=e)
        p.f = f.reshape(-1).copy()
        u, rep = solver.solve(p, default_options(method=abi.JACOBI, max_iter=1, tol=0.0))
        with np.errstate(all="ignore"):
            ref = (-f - 0.0) / e
        assert same(u.reshape(NY, NX)[1:-1, 1:-1], ref[1:-1, 1:-1]), e


@pytest.mark.parametrize("seed, lo, hi", [(4, -1074, 1000), (5, -650, 650)])
def test_heat_quotients(seed, lo, hi):
    f = dividends(seed, lo, hi)
    for ut in divisors(seed):
        p = GridProblem(NX, NY, 1, ut=ut)
        p.f = f.reshape(-1).copy()
        u, rep = solver.time_series(p, 0.0, 1.0, 5, frame_stride=4)
        with np.errstate(all="ignore"):
            q = -(0.0 + f) / ut
            q[~np.isfinite(q)] = 0.0
            ref = np.zeros_like(f)
            for _ in range(4):
                ref = ref + q
        # (a sum that overflows makes NaN of itself and its neighbours through the operator's zero weights)
        fin = np.pad(np.isfinite(ref), 1, constant_values=True)
        ok = (fin[1:-1, 1:-1] & fin[2:, 1:-1] & fin[:-2, 1:-1] & fin[1:-1, 2:] & fin[1:-1, :-2])[1:-1, 1:-1]
        assert ok.mean() > 0.99
        assert same(u.reshape(NY, NX)[1:-1, 1:-1][ok], ref[1:-1, 1:-1][ok]), ut
