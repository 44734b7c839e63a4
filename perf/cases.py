"""Performance cases of the solve library: what its users run, through its public Python entry points.

The cases cover the reference methods (CG, Jacobi, SOR, BiCGStab) at the small sizes they are used at, the
multigrid-preconditioned solves from small ragged grids to 257^3 and 513^3 in FP64 and in FP32-inside-FP64
refinement, explicit heat runs, the pressure projection, and a batch of many uneven grids. Inputs are made on
the GPU from a seed, in the shapes and distributions of `pde_solver_b200.synthetic`.
"""
import math

import numpy as np
import torch

from pde_solver_b200 import abi, solver
from pde_solver_b200.batch import Batch
from pde_solver_b200.problem import FaceBC, GridProblem, default_options

DEV = "cuda"

# Face sets by name: (left, right, bottom, top, front, back), each (kind, value...) with
# D = Dirichlet value, N = Neumann slope, R = Robin alpha, beta, gamma.
FACES = {
    "dirichlet": ["D0"] * 6,
    # the headline workload's faces: Robin on a min face
    "headline": ["D0", "D0", "N0", "N0", "R1,1,0", "D0"],
    # every closure kind, non-zero data
    "mixed": ["R1,0.5,0.2", "D0", "N0.3", "D1", "N0.1", "D0.5"],
}

METHODS = {"cg": abi.CG, "jacobi": abi.JACOBI, "sor": abi.SOR, "bicgstab": abi.BICGSTAB, "mgpcg": abi.MG_PCG,
           "mgbicgstab": abi.MG_BICGSTAB}


def _solve_case(name, method, nx, ny, nz, coef, faces="dirichlet", tol=1e-10, relative=True, max_iter=1000,
                precision="fp64", mem="device"):
    c = dict(kind="solve", method=method, nx=nx, ny=ny, nz=nz, coef=coef, faces=faces, tol=tol, relative=relative,
             max_iter=max_iter, precision=precision, mem=mem)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: CG on the manufactured-solution grid of the test suite, a handful of iterations
        _solve_case("cg_129x129", "cg", 129, 129, 1, "poisson"),
        # the default method with its default tolerance: many cheap sweeps on a small grid
        _solve_case("jacobi_129x129", "jacobi", 129, 129, 1, "poisson", tol=1e-6, relative=False, max_iter=50000),
        # SOR in the reference's lexicographic order, every boundary kind, ragged sides
        _solve_case("sor_97x65_mixed", "sor", 97, 65, 1, "poisson", "mixed", tol=1e-6, relative=False,
                    max_iter=20000),
        # per-node coefficients with convection: the Krylov method users take for nonsymmetric operators
        _solve_case("bicgstab_97x81_nodal", "bicgstab", 97, 81, 1, "nodal", tol=1e-8, max_iter=4000),
        # a 2D request of the serving mix
        _solve_case("mgpcg_257x193", "mgpcg", 257, 193, 1, "divk_rough"),
        # ragged 3D grid: even sides (non-nested levels), every boundary kind
        _solve_case("mgpcg_100x77x58_mixed", "mgpcg", 100, 77, 58, "divk_rough", "mixed"),
        # the headline: variable-coefficient Poisson in FP64
        _solve_case("mgpcg_257", "mgpcg", 257, 257, 257, "divk", "headline"),
        # host arrays in and out, FP32 refinement with BF16 smoother coefficients: the drop-in caller's way
        _solve_case("mixed_bf16_129_host", "mgpcg", 129, 129, 129, "divk", "headline", precision="bf16", mem="host"),
        # the largest call: convection-diffusion in mixed precision
        _solve_case("convdiff_513_mixed", "mgbicgstab", 513, 513, 513, "convdiff", precision="mixed"),
        # 200 explicit heat steps with a few frames shown, as the serving mix runs them
        dict(name="heat_257x257_200", kind="heat", nx=257, ny=257, nz=1, steps=200, frame_stride=50),
        # one pressure projection of a random velocity field
        dict(name="projection_256x256", kind="projection", nx=256, ny=256, tol=1e-10),
        # one group of uneven grids, 2D and 3D in the batched workload's proportion
        dict(name="batch_56x2d_8x3d", kind="batch", n2d=56, n3d=8, lo2=33, hi2=513, lo3=17, hi3=129),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cg", "jacobi", "sor", "bicgstab", "mgpcg2", "mgpcg3", "mgpcg3", "convdiff", "heat",
                       "projection", "batch"])
    if kind == "cg":
        n = _logint(rng, 33, 513)
        return _solve_case("", "cg", n, max(17, int(n * rng.uniform(0.5, 1.0))), 1, "poisson")
    if kind in ("jacobi", "sor"):
        faces = rng.choice(["dirichlet", "mixed"])
        it = 50000 if kind == "jacobi" else 20000
        if rng.random() < 0.3:
            n = _logint(rng, 9, 33)
            return _solve_case("", kind, n, max(5, int(n * rng.uniform(0.6, 1.0))), max(5, int(n * rng.uniform(0.6, 1.0))),
                               "poisson", faces, tol=1e-6, relative=False, max_iter=it)
        n = _logint(rng, 17, 129 if kind == "jacobi" else 97)
        return _solve_case("", kind, n, max(9, int(n * rng.uniform(0.5, 1.0))), 1, "poisson", faces, tol=1e-6,
                           relative=False, max_iter=it)
    if kind == "bicgstab":
        n = _logint(rng, 25, 161)
        return _solve_case("", "bicgstab", n, max(17, int(n * rng.uniform(0.6, 1.0))), 1, "nodal", tol=1e-8,
                           max_iter=4000)
    if kind == "mgpcg2":
        n = _logint(rng, 33, 1025)
        return _solve_case("", "mgpcg", n, max(17, int(n * rng.uniform(0.6, 1.0))), 1, "divk_rough",
                           rng.choice(list(FACES)), precision=rng.choice(["fp64", "mixed"]))
    if kind == "mgpcg3":
        n = _logint(rng, 17, 257)
        side = lambda: max(9, int(n * rng.uniform(0.6, 1.0)))  # noqa: E731
        dims = (n, n, n) if rng.random() < 0.4 else (n, side(), side())
        return _solve_case("", "mgpcg", *dims, rng.choice(["divk", "divk_rough", "poisson"]), rng.choice(list(FACES)),
                           precision=rng.choice(["fp64", "fp64", "mixed", "bf16"]),
                           mem=rng.choice(["device", "device", "host"]))
    if kind == "convdiff":
        n = _logint(rng, 33, 385)
        return _solve_case("", "mgbicgstab", n, n, n, "convdiff", precision=rng.choice(["fp64", "mixed"]))
    if kind == "heat":
        if rng.random() < 0.3:
            n = _logint(rng, 17, 97)
            return dict(kind="heat", nx=n, ny=n, nz=n, steps=rng.randrange(50, 201), frame_stride=50)
        n = _logint(rng, 65, 513)
        return dict(kind="heat", nx=n, ny=max(33, int(n * rng.uniform(0.5, 1.0))), nz=1, steps=rng.randrange(50, 201),
                    frame_stride=rng.choice([10, 50, 1000]))
    if kind == "projection":
        n = _logint(rng, 64, 513)
        return dict(kind="projection", nx=n, ny=max(33, int(n * rng.uniform(0.6, 1.0))), tol=1e-10)
    return dict(kind="batch", n2d=rng.randrange(1, 57), n3d=rng.randrange(0, 9), lo2=33, hi2=513, lo3=17,
                hi3=rng.randrange(33, 130))


# ------------------------------------------------------------------ inputs


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _randn(shape, g):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float64)


def _smooth(a, passes=3):
    """`passes` 3^d box averages with replicated borders."""
    dim = a.dim()
    x = a[None, None]
    pad = (1, 1) * dim
    pool = torch.nn.functional.avg_pool3d if dim == 3 else torch.nn.functional.avg_pool2d
    for _ in range(passes):
        x = pool(torch.nn.functional.pad(x, pad, mode="replicate"), 3, stride=1)
    return x[0, 0].contiguous()


def _spacing(nx, ny, nz):
    return 1.0 / (nx - 1), 1.0 / (ny - 1), (1.0 / (nz - 1) if nz > 1 else 0.0)


def _modes(nx, ny, nz, g, count=5):
    """A seeded sum of smooth sine modes, the right sides of manufactured solutions."""
    amp = _randn((count,), g).tolist()
    ax = [torch.linspace(0.0, 1.0, m, dtype=torch.float64, device=DEV) for m in (nz, ny, nx)]
    f = torch.zeros((nz, ny, nx), dtype=torch.float64, device=DEV)
    for q, a in enumerate(amp):
        kx, ky, kz = 1 + q % 2, 1 + (q // 2) % 2, 1 + q // 4
        t = torch.sin(math.pi * ky * ax[1])[:, None] * torch.sin(math.pi * kx * ax[2])[None, :]
        z = torch.sin(math.pi * kz * ax[0]) if nz > 1 else torch.ones(1, dtype=torch.float64, device=DEV)
        f += (2.0 + a) * math.pi ** 2 * (kx * kx + ky * ky) * z[:, None, None] * t[None]
    return -f


def _fields(c, seed):
    """The arrays and scalars of a steady problem: dict with f, and k or nodal or constants."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    shape = (nz, ny, nx)
    g = _gen(seed)
    d = dict(a=0.0, b=0.0, az=0.0, c=0.0, d=0.0, dz=0.0, e=0.0, k=None, nodal=None)
    if c["coef"] == "poisson":
        d.update(a=-1.0, b=-1.0, az=-1.0 if nz > 1 else 0.0)
        d["f"] = _randn(shape, g) if c["method"] == "mgpcg" else _modes(nx, ny, nz, g)
    elif c["coef"] in ("divk", "divk_rough"):
        if c["coef"] == "divk":  # log-normal, sigma 1, three box passes
            e = torch.exp(_randn(shape, g))
            d["k"] = _smooth(e if nz > 1 else e[0]).reshape(shape)
        else:  # log-normal, sigma 0.5, independent per node
            d["k"] = torch.exp(0.5 * _randn(shape, g))
        d["f"] = -_randn(shape, g)
    elif c["coef"] == "convdiff":  # -eps Laplace(u) + b.grad(u), b a seeded unit vector
        bv = torch.randn(3, generator=torch.Generator().manual_seed(int(seed) & 0x7FFFFFFF), dtype=torch.float64)
        bv = (bv / bv.norm()).tolist()
        d.update(a=-1e-2, b=-1e-2, az=-1e-2, c=bv[0], d=bv[1], dz=bv[2])
        d["f"] = -(2.0 * torch.rand(shape, generator=g, device=DEV, dtype=torch.float64) - 1.0)
    else:  # nodal: a, b, az, c, d, dz, e arrays
        y = torch.linspace(0.0, 1.0, ny, dtype=torch.float64, device=DEV)[:, None].expand(ny, nx)
        x = torch.linspace(0.0, 1.0, nx, dtype=torch.float64, device=DEV)[None, :].expand(ny, nx)
        zero = torch.zeros_like(x)
        w = _randn((3,), g).abs().tolist()
        d["nodal"] = torch.stack([-(1.0 + w[0] * x * y), -(1.5 + torch.sin(3.0 * x)), zero, w[1] * x, -w[2] * y, zero,
                                  zero - 0.1]).reshape(7, nz, ny, nx).contiguous()
        d["f"] = _modes(nx, ny, nz, g)
    return d


def _faces(name):
    out = []
    for s in FACES[name]:
        v = [float(t) for t in s[1:].split(",")]
        out.append({"D": FaceBC.dirichlet, "N": FaceBC.neumann, "R": FaceBC.robin}[s[0]](*v))
    return out


def _host(t):
    h = torch.empty(t.numel(), dtype=torch.float64, pin_memory=True)
    h.copy_(t.reshape(-1))
    return h.numpy()


def _heat_dt(c):
    hx, hy, hz = _spacing(c["nx"], c["ny"], c["nz"])
    return 0.9 / (2.0 * (1.0 / hx ** 2 + 1.0 / hy ** 2 + (1.0 / hz ** 2 if c["nz"] > 1 else 0.0)))


def _heat_u0(c, seed):
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    g = _gen(seed)
    cx, cy, cz, w = (0.4 + 0.2 * torch.rand(4, generator=g, device=DEV, dtype=torch.float64)).tolist()
    ax = [torch.linspace(0.0, 1.0, m, dtype=torch.float64, device=DEV) for m in (nx, ny)]
    r2 = (ax[0][None, None, :] - cx) ** 2 + (ax[1][None, :, None] - cy) ** 2
    if nz > 1:
        r2 = r2 + (torch.linspace(0.0, 1.0, nz, dtype=torch.float64, device=DEV)[:, None, None] - cz) ** 2
    return torch.exp(-(20.0 + 40.0 * w) * r2).contiguous()


def _members(c, seed):
    """Sides and fields of a batch: (nx, ny, nz, k, f) per member, k log-normal sigma 0.5, f Gaussian. The sides
    are part of the case (quantiles of the log-uniform ranges), the fields come from the seed."""
    out = []
    g = _gen(seed)
    for cnt, lo, hi, is3 in ((c["n2d"], c["lo2"], c["hi2"], False), (c["n3d"], c["lo3"], c["hi3"], True)):
        for q in range(cnt):
            n = int(round(math.exp(math.log(lo) + (q + 0.5) / cnt * (math.log(hi) - math.log(lo)))))
            shape = (n, n, n) if is3 else (1, n, n)
            out.append((n, n, n if is3 else 1, torch.exp(0.5 * _randn(shape, g)), -_randn(shape, g)))
    return out


def prepare(case, seed):
    c = case
    if c["kind"] == "solve":
        d = _fields(c, seed)
        p = GridProblem(c["nx"], c["ny"], c["nz"], a=d["a"], b=d["b"], az=d["az"], c=d["c"], d=d["d"], dz=d["dz"],
                        e=d["e"], faces=_faces(c["faces"]))
        p.coef_kind = abi.COEF_DIVK if d["k"] is not None else abi.COEF_NODAL if d["nodal"] is not None else abi.COEF_CONST
        opt = default_options(method=METHODS[c["method"]], tol=c["tol"], max_iter=c["max_iter"],
                              tol_mode=abi.TOL_RELATIVE if c["relative"] else abi.TOL_REFERENCE,
                              precision=abi.FP64 if c["precision"] == "fp64" else abi.MIXED,
                              bf16_coefficients=1 if c["precision"] == "bf16" else 0)
        s = dict(kind="solve", mem=c["mem"], problem=p, options=opt)
        if c["mem"] == "host":
            p.f, p.k = _host(d["f"]), (_host(d["k"]) if d["k"] is not None else None)
            p.nodal = _host(d["nodal"]) if d["nodal"] is not None else None
            s["out"] = torch.empty(p.n, dtype=torch.float64, pin_memory=True).numpy()
        else:
            p.mem_space = abi.MEM_DEVICE
            s["fields"] = d  # keeps the device arrays alive
            p.f_dev = d["f"].data_ptr()
            p.k_dev = d["k"].data_ptr() if d["k"] is not None else 0
            p.nodal_dev = d["nodal"].data_ptr() if d["nodal"] is not None else 0
            s["out"] = torch.empty(p.n, dtype=torch.float64, device=DEV)
        return s
    if c["kind"] == "heat":
        p = GridProblem(c["nx"], c["ny"], c["nz"], a=-1.0, b=-1.0, az=-1.0 if c["nz"] > 1 else 0.0, ut=1.0)
        p.u0 = _heat_u0(c, seed).reshape(-1).cpu().numpy()
        return dict(kind="heat", problem=p, dt=_heat_dt(c), steps=c["steps"], frame_stride=c["frame_stride"])
    if c["kind"] == "projection":
        g = _gen(seed)
        n = c["nx"] * c["ny"]
        return dict(kind="projection", case=dict(c), u=_randn((n,), g).cpu().numpy(), v=_randn((n,), g).cpu().numpy(),
                    p=np.zeros(n))
    probs, keep = [], []
    for nx, ny, nz, k, f in _members(c, seed):
        probs.append(GridProblem(nx, ny, nz, coef_kind=abi.COEF_DIVK, mem_space=abi.MEM_DEVICE, k_dev=k.data_ptr(),
                                 f_dev=f.data_ptr()))
        keep.append((k, f))
    torch.cuda.synchronize()
    b = Batch(probs)
    rhs = torch.cat([f.reshape(-1) for _, f in keep])
    torch.cuda.synchronize()
    return dict(kind="batch", batch=b, keep=keep, rhs=rhs,
                out=torch.empty(b.nodes, dtype=torch.float64, pin_memory=True).numpy())


def run(state):
    s = state
    if s["kind"] == "solve":
        if s["mem"] == "host":
            u, _ = solver.solve(s["problem"], s["options"], out=s["out"])
            return u
        solver.solve(s["problem"], s["options"], out=s["out"].data_ptr())
        return s["out"]
    if s["kind"] == "heat":
        frames = []
        u, _ = solver.time_series(s["problem"], 0.0, s["dt"], s["steps"] + 1,
                                  on_frame=lambda q, t, grid: frames.append(grid), frame_stride=s["frame_stride"])
        return {"u": u, "frames": frames}
    if s["kind"] == "projection":
        c = s["case"]
        u, v, _, p, _ = solver.project_velocity(s["u"], s["v"], None, s["p"], c["nx"], c["ny"], 1, 1.0 / (c["nx"] - 1),
                                                1.0 / (c["ny"] - 1), 1.0, 0.01, 20000, c["tol"])
        return u, v, p
    b = s["batch"]
    b.load_rhs(s["rhs"].data_ptr(), abi.MEM_DEVICE)
    b.solve(1e-10)
    return b.read_packed(s["out"])


def work(case):
    """Each input field read once and each result written once; one residual evaluation's arithmetic."""
    c = case
    if c["kind"] == "solve":
        n = c["nx"] * c["ny"] * c["nz"]
        arrays = 2 + (1 if c["coef"].startswith("divk") else 7 if c["coef"] == "nodal" else 0)
        return {"bytes": 8.0 * n * arrays, "flops": 20.0 * n}
    if c["kind"] == "heat":
        n = c["nx"] * c["ny"] * c["nz"]
        shown = len([q for q in range(c["steps"] + 1) if q % c["frame_stride"] == 0 or q == c["steps"]])
        return {"bytes": 8.0 * n * (2 + shown), "flops": 15.0 * n * c["steps"]}
    if c["kind"] == "projection":
        n = c["nx"] * c["ny"]
        return {"bytes": 8.0 * n * 6, "flops": 30.0 * n}
    n = 0
    for cnt, lo, hi, dim in ((c["n2d"], c["lo2"], c["hi2"], 2), (c["n3d"], c["lo3"], c["hi3"], 3)):
        for q in range(cnt):
            n += int(round(math.exp(math.log(lo) + (q + 0.5) / cnt * (math.log(hi) - math.log(lo))))) ** dim
    return {"bytes": 8.0 * n * 3, "flops": 20.0 * n}


# ------------------------------------------- 64-bit values in plain torch


class _System:
    """The discrete equations on a (nz, ny, nx) grid: weights per interior node, boundary closures."""

    def __init__(self, nx, ny, nz, d, faces):
        self.nx, self.ny, self.nz, self.is3 = nx, ny, nz, nz > 1
        hx, hy, hz = _spacing(nx, ny, nz)
        self.h = (hx, hx, hy, hy, hz, hz)
        self.face = []
        for s in FACES[faces]:
            self.face.append((s[0], [float(t) for t in s[1:].split(",")]))
        self.K = slice(1, -1) if self.is3 else slice(None)
        inner = (self.K, slice(1, -1), slice(1, -1))
        if d["k"] is not None:
            k = d["k"]
            nb = self._neighbours(k)
            kc = k[inner]
            w = [-0.5 * (kc + q) for q in nb]
            hh = (hx, hx, hy, hy, hz, hz)
            self.w = [w[q] / hh[q] ** 2 for q in range(len(w))]
            self.center = -sum(self.w)
        else:
            if d["nodal"] is not None:
                a, b, az, cc, dd, dz, e = (t[inner] for t in d["nodal"])
            else:
                a, b, az, cc, dd, dz, e = (torch.tensor(d[q], dtype=torch.float64, device=DEV)
                                           for q in ("a", "b", "az", "c", "d", "dz", "e"))
            ax, by, cx, cy = a / hx ** 2, b / hy ** 2, cc / (2 * hx), dd / (2 * hy)
            self.w = [ax - cx, ax + cx, by - cy, by + cy]
            self.center = -2 * ax - 2 * by + e
            if self.is3:
                bz, cz = az / hz ** 2, dz / (2 * hz)
                self.w += [bz - cz, bz + cz]
                self.center = self.center - 2 * bz
        self.inner = inner
        self.f = d.get("f")

    def _neighbours(self, u):
        K, I, lo, hi = self.K, slice(1, -1), slice(0, -2), slice(2, None)
        out = [u[K, I, lo], u[K, I, hi], u[K, lo, I], u[K, hi, I]]
        return out + [u[lo, I, I], u[hi, I, I]] if self.is3 else out

    def _where(self, q, at):
        """The plane of face q itself (at=0) or next to it (at=1)."""
        s = [slice(None)] * 3
        s[2 - q // 2] = at if q % 2 == 0 else -1 - at
        return tuple(s)

    def close(self, u, homogeneous=False):
        """Boundary values of u in place: x, y, z closures, then Dirichlet."""
        for q in range(6 if self.is3 else 4):
            kind, v = self.face[q]
            h, nxt = self.h[q], u[self._where(q, 1)]
            if kind == "N":
                s = 0.0 if homogeneous else v[0]
                u[self._where(q, 0)] = nxt - h * s if q % 2 == 0 else nxt + h * s
            elif kind == "R":
                al, be, ga = v
                ga = 0.0 if homogeneous else ga
                u[self._where(q, 0)] = ((ga + be / h * nxt) / (al + be / h) if q % 2 == 0
                                        else (ga - be / h * nxt) / (al - be / h))
        for q in range(6 if self.is3 else 4):
            if self.face[q][0] == "D":
                u[self._where(q, 0)] = 0.0 if homogeneous else self.face[q][1][0]
        return u

    def neighbour_sum(self, u):
        nb = self._neighbours(u)
        t = self.w[0] * nb[0]
        for q in range(1, len(nb)):
            t = t + self.w[q] * nb[q]
        return t

    def full(self, v):
        u = torch.zeros((self.nz, self.ny, self.nx), dtype=torch.float64, device=DEV)
        u[self.inner] = v
        return u

    def apply(self, v, homogeneous=True):
        u = self.close(self.full(v), homogeneous)
        return self.center * v + self.neighbour_sum(u)

    def solve(self, symmetric, rel=1e-13, max_iter=20000):
        zero = torch.zeros_like(self.f[self.inner])
        b = -self.f[self.inner] - self.apply(zero, False)
        ones = torch.ones_like(zero)
        # the folded diagonal: the closure factor of a face stands beside the node next to it
        diag = self.center * ones
        for q in range(6 if self.is3 else 4):
            kind, v = self.face[q]
            h = self.h[q]
            c1 = 1.0 if kind == "N" else 0.0
            if kind == "R":
                c1 = (v[1] / h) / (v[0] + v[1] / h) if q % 2 == 0 else (-v[1] / h) / (v[0] - v[1] / h)
            if c1:
                s = [slice(None)] * 3
                s[2 - q // 2] = 0 if q % 2 == 0 else -1
                diag[tuple(s)] += c1 * (self.w[q] * ones)[tuple(s)]
        x, r = zero, b
        stop = rel * float(b.norm())
        dot = lambda p, q: (p * q).sum()  # noqa: E731
        if symmetric:
            z = r / diag
            p, rz = z, dot(r, z)
            for it in range(max_iter):
                q = self.apply(p)
                al = rz / dot(p, q)
                x, r = x + al * p, r - al * q
                if it % 20 == 19 and float(r.norm()) <= stop:
                    break
                z = r / diag
                new = dot(r, z)
                p, rz = z + (new / rz) * p, new
        else:
            rh, p, v = r, r, None
            rho = dot(rh, r)
            for it in range(max_iter):
                ph = p / diag
                v = self.apply(ph)
                al = rho / dot(rh, v)
                s = r - al * v
                sh = s / diag
                t = self.apply(sh)
                om = dot(t, s) / dot(t, t)
                x, r = x + al * ph + om * sh, s - om * t
                if it % 10 == 9 and float(r.norm()) <= stop:
                    break
                new = dot(rh, r)
                p = r + (new / rho) * (al / om) * (p - om * v)
                rho = new
        return self.close(self.full(x))

    def jacobi(self, tol, max_iter):
        """The Jacobi method itself: the same sweeps, the same stopping rule."""
        u = self.close(torch.zeros((self.nz, self.ny, self.nx), dtype=torch.float64, device=DEV))
        f = self.f[self.inner]
        group, done = 32, 0
        while done < max_iter:
            m, kept, delta = min(group, max_iter - done), [], []
            for _ in range(m):
                new = (-f - self.neighbour_sum(u)) / self.center
                delta.append((new - u[self.inner]).abs().max())
                u = self.close(self.full(new))
                kept.append(u)
            done += m
            for q, v in enumerate(torch.stack(delta).tolist()):
                if v < tol:
                    return kept[q]
        return u


def _exact_projection(c, s):
    nx, ny = c["nx"], c["ny"]
    hx, hy, dt = 1.0 / (nx - 1), 1.0 / (ny - 1), 0.01
    u = torch.from_numpy(s["u"]).to(DEV).reshape(ny, nx)
    v = torch.from_numpy(s["v"]).to(DEV).reshape(ny, nx)

    def grad(a, h, dim):
        a = a.movedim(dim, 0)
        g = torch.empty_like(a)
        g[1:-1] = (a[2:] - a[:-2]) / (2 * h)
        g[0], g[-1] = (a[1] - a[0]) / h, (a[-1] - a[-2]) / h
        return g.movedim(0, dim)

    def cosines(n):
        i = torch.arange(n, dtype=torch.float64, device=DEV)
        m = torch.cos(math.pi / n * i[:, None] * (i[None, :] + 0.5)) * math.sqrt(2.0 / n)
        m[0] /= math.sqrt(2.0)
        return m, 2.0 * torch.cos(math.pi / n * i) - 2.0

    rhs = (grad(u, hx, 1) + grad(v, hy, 0)) / dt
    (cx, lx), (cy, ly) = cosines(nx), cosines(ny)
    t = cy @ (rhs - rhs.mean()) @ cx.T
    lam = ly[:, None] / hy ** 2 + lx[None, :] / hx ** 2
    lam[0, 0] = 1.0
    t = t / lam
    t[0, 0] = 0.0
    p = cy.T @ t @ cx
    return (u - dt * grad(p, hx, 1)).reshape(-1), (v - dt * grad(p, hy, 0)).reshape(-1), p.reshape(-1)


def exact(case, seed):
    c = case
    if c["kind"] == "solve":
        n = c["nx"] * c["ny"] * c["nz"]
        if c["coef"] == "convdiff" and n > 200 ** 3:
            return None
        d = _fields(c, seed)
        sys_ = _System(c["nx"], c["ny"], c["nz"], d, c["faces"])
        if c["method"] == "jacobi":
            return sys_.jacobi(c["tol"], c["max_iter"]).reshape(-1)
        return sys_.solve(c["coef"] in ("poisson", "divk", "divk_rough")).reshape(-1)
    if c["kind"] == "heat":
        u = _heat_u0(c, seed)
        d = dict(a=-1.0, b=-1.0, az=-1.0 if c["nz"] > 1 else 0.0, c=0.0, d=0.0, dz=0.0, e=0.0, k=None, nodal=None)
        sys_ = _System(c["nx"], c["ny"], c["nz"], d, "dirichlet")
        u = sys_.close(u.clone())
        dt, frames = _heat_dt(c), []
        for q in range(c["steps"] + 1):
            if q % c["frame_stride"] == 0 or q == c["steps"]:
                frames.append(u.reshape(-1).clone())
            if q < c["steps"]:
                v = u[sys_.inner]
                u = sys_.close(sys_.full(v - dt * (sys_.center * v + sys_.neighbour_sum(u))))
        return {"u": u.reshape(-1), "frames": frames}
    if c["kind"] == "projection":
        return _exact_projection(c, prepare(c, seed))
    out = []
    for nx, ny, nz, k, f in _members(c, seed):
        d = dict(a=0.0, b=0.0, az=0.0, c=0.0, d=0.0, dz=0.0, e=0.0, k=k, nodal=None, f=f)
        out.append(_System(nx, ny, nz, d, "dirichlet").solve(True).reshape(-1))
    return torch.cat(out)
