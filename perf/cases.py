"""Performance cases of the solver library: what a user of it runs, over the
range of sizes it is used at.

A program that uses the library keeps one mesh for thousands of time steps.
Every step brings new coefficients and a new source and asks for a solve; so
a pass stages the coefficients and solves from psi = 0.  The mesh
(addressing, context) is what the program keeps, and its cell numbering does
not depend on the seed; coefficients and sources do.

Kinds of case
  spmv      y = A x and w.y on the caller's own device arrays, the call of
            programs that may not allocate (cf_ldu_spmv_dot_noalloc)
  pressure  cudaPCG on a symmetric pressure matrix, device arrays
  momentum  cudaPBiCGStab on an upwind convection-diffusion matrix, one
            component or three that share the matrix
  batch     many independent pressure systems of uneven sizes at once
  adjoint   a solve, then the gradients of 0.5 |x - x*|^2 with respect to
            b, diag, upper and lower

"host" cases go through the lduMatrix::solver surface with numpy arrays, as
an OpenFOAM-like program does; the others keep everything on the GPU.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from metal4foam_b200 import _lib, mesh
from metal4foam_b200.solver import lduAddressing, lduMatrix

DEV = "cuda:0"

# options of the solves by kind (the rest are the library's defaults)
OPTIONS = {
    "pressure": dict(tolerance=1e-6, maxIter=5000),
    "momentum": dict(maxIter=5000),
    "batch": dict(tolerance=1e-6, stagnationLimit=400, maxRestarts=20, maxIter=20000),
    "adjoint": dict(tolerance=1e-10, maxRestarts=12, maxIter=5000),
}


def listed():
    return [
        # the smallest call: one product on a mesh of one processor's share,
        # latency counts
        dict(name="spmv_40x37x33", kind="spmv", mesh="grid", nx=40, ny=37, nz=33, permute=False,
             symmetric=True),
        # 2-D Poisson 128^2: the plain small solve every OpenFOAM tutorial has
        dict(name="pcg_poisson_128x128", kind="pressure", mesh="grid", nx=128, ny=128, nz=1,
             permute=False, coeffs="poisson", order=4, precond="Chebyshev", host=False),
        # a small 3-D pressure solve through the solver surface, host arrays
        dict(name="pcg_host_31x29x27", kind="pressure", mesh="grid", nx=31, ny=29, nz=27,
             permute=False, coeffs="varcoeff", order=8, precond="Chebyshev", host=True),
        # a small momentum solve through the solver surface, host arrays
        dict(name="bicg_host_25x23x21", kind="momentum", nx=25, ny=23, nz=21, nrhs=1, tol=1e-6,
             host=True),
        # an ordinary 2-D case
        dict(name="pcg_poisson_640x480", kind="pressure", mesh="grid", nx=640, ny=480, nz=1,
             permute=False, coeffs="poisson", order=8, precond="Chebyshev", host=False),
        # an ordinary mesh of prisms (five neighbours) in scattered numbering
        dict(name="pcg_prism_61x53x31", kind="pressure", mesh="prism", nx=61, ny=53, nz=31,
             permute=True, coeffs="varcoeff", order=8, precond="Chebyshev", host=False),
        # the headline: 128^3 variable-coefficient pressure, permuted cells
        dict(name="pcg_128x128x128", kind="pressure", mesh="grid", nx=128, ny=128, nz=128,
             permute=True, coeffs="varcoeff", order=8, precond="Chebyshev", host=False),
        # a large pressure solve with the multigrid preconditioner, odd sizes
        dict(name="gamg_101x97x89", kind="pressure", mesh="grid", nx=101, ny=97, nz=89,
             permute=True, coeffs="varcoeff", order=8, precond="GAMG", host=False),
        # the large momentum solve, one component, tight tolerance
        dict(name="bicg_96x96x96", kind="momentum", nx=96, ny=96, nz=96, nrhs=1, tol=1e-8,
             host=False),
        # Ux, Uy, Uz on one matrix
        dict(name="bicg_64x64x64_3rhs", kind="momentum", nx=64, ny=64, nz=64, nrhs=3, tol=1e-6,
             host=False),
        # many uneven systems together
        dict(name="batch_16", kind="batch", count=16, nmin=1000, nmax=100000, shape=3),
        # gradients through a solve
        dict(name="adjoint_64x60x56", kind="adjoint", nx=64, ny=60, nz=56, permute=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims3(rng, cells):
    base = cells ** (1.0 / 3.0)
    nx = max(3, int(round(base * 2.0 ** rng.uniform(-0.4, 0.4))))
    ny = max(3, int(round(base * 2.0 ** rng.uniform(-0.4, 0.4))))
    return nx, ny, max(3, int(round(cells / (nx * ny))))


def _dims2(rng, cells):
    nx = max(8, int(round(math.sqrt(cells * 2.0 ** rng.uniform(-1.0, 1.0)))))
    return nx, max(8, int(round(cells / nx))), 1


def draw(rng):
    """One more case of the listed kinds' ranges."""
    kind = rng.choice(["spmv", "pressure3", "pressure3", "pressure2", "prism", "gamg", "momentum",
                       "momentum", "batch", "adjoint"])
    if kind == "spmv":
        nx, ny, nz = _dims3(rng, _log_int(rng, 2000, 1000000))
        return dict(kind="spmv", mesh="grid", nx=nx, ny=ny, nz=nz, permute=rng.random() < 0.3,
                    symmetric=rng.random() < 0.5)
    if kind == "pressure3":
        nx, ny, nz = _dims3(rng, _log_int(rng, 2000, 1900000))
        return dict(kind="pressure", mesh="grid", nx=nx, ny=ny, nz=nz, permute=rng.random() < 0.5,
                    coeffs="varcoeff", order=rng.choice([4, 8, 8]), precond="Chebyshev",
                    host=rng.random() < 0.3)
    if kind == "pressure2":
        nx, ny, nz = _dims2(rng, _log_int(rng, 2000, 350000))
        return dict(kind="pressure", mesh="grid", nx=nx, ny=ny, nz=nz, permute=rng.random() < 0.3,
                    coeffs="poisson", order=rng.choice([4, 8]), precond="Chebyshev", host=False)
    if kind == "prism":
        nx, ny, nz = _dims3(rng, _log_int(rng, 2000, 300000))
        return dict(kind="pressure", mesh="prism", nx=nx, ny=ny, nz=nz, permute=True,
                    coeffs="varcoeff", order=8, precond="Chebyshev", host=False)
    if kind == "gamg":
        nx, ny, nz = _dims3(rng, _log_int(rng, 20000, 900000))
        return dict(kind="pressure", mesh="grid", nx=nx, ny=ny, nz=nz, permute=rng.random() < 0.5,
                    coeffs="varcoeff", order=8, precond="GAMG", host=False)
    if kind == "momentum":
        nrhs = rng.choice([1, 3])
        nx, ny, nz = _dims3(rng, _log_int(rng, 2000, 900000 if nrhs == 1 else 300000))
        return dict(kind="momentum", nx=nx, ny=ny, nz=nz, nrhs=nrhs,
                    tol=rng.choice([1e-6, 1e-8]), host=rng.random() < 0.3)
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(6, 16), nmin=1000, nmax=100000,
                    shape=rng.randint(4, 1 << 20))
    nx, ny, nz = _dims3(rng, _log_int(rng, 4000, 260000))
    return dict(kind="adjoint", nx=nx, ny=ny, nz=nz, permute=rng.random() < 0.5)


# ------------------------------------------------------------------- meshes


class _Mesh:
    """A mesh in a fixed cell numbering: addressing plus, for grids in their
    natural numbering, the direction of every face."""

    def __init__(self, addr, axis, dims):
        self.addr = addr
        self.axis = axis
        self.dims = dims
        self.ldu = lduAddressing(addr)     # what a program using the surface keeps
        self.n, self.nf = addr.n, addr.nf


@functools.lru_cache(maxsize=12)
def _mesh(kind, nx, ny, nz, permute):
    dims = (nx, ny) if kind == "grid" and nz == 1 else (nx, ny, nz)
    axis = None
    if kind == "prism":
        low, upp = mesh.prism_faces(nx, ny, nz)
        n = 2 * nx * ny * nz
    else:
        low, upp, axis = mesh.structured_faces(dims)
        n = nx * ny * nz
    if permute:
        label = np.random.default_rng(n).permutation(n).astype(np.int64)
        low, upp = mesh.permute_cells(label, low, upp)
        axis = None
    return _Mesh(mesh.ldu_addressing(n, low, upp), axis, dims)


def _batch_dims(case):
    """Cell counts log-uniform between nmin and nmax, every other system 2-D."""
    rng = np.random.default_rng(case["shape"])
    out = []
    for s in range(case["count"]):
        cells = math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"])))
        if s % 2 == 0:
            nx = max(2, int(round(math.sqrt(cells * 2.0 ** rng.uniform(-1.0, 1.0)))))
            out.append((nx, max(2, int(round(cells / nx))), 1))
        else:
            base = cells ** (1.0 / 3.0)
            nx = max(2, int(round(base * 2.0 ** rng.uniform(-0.5, 0.5))))
            ny = max(2, int(round(base * 2.0 ** rng.uniform(-0.5, 0.5))))
            out.append((nx, ny, max(2, int(round(cells / (nx * ny))))))
    return out


# --------------------------------------------------------------- coefficients


def _diag_of(m, upper, lower):
    return -(np.bincount(m.addr.lowerAddr, weights=upper, minlength=m.n)
             + np.bincount(m.addr.upperAddr, weights=lower, minlength=m.n))


def _pressure_system(m, coeffs, seed):
    """Poisson (-1 per face) or log-uniform conductivities over four decades
    with harmonic means on the faces; Neumann boundaries, reference cell 0;
    source ~ N(0,1) with zero mean."""
    rng = np.random.default_rng(seed)
    a = m.addr
    if coeffs == "poisson":
        upper = np.full(m.nf, -1.0)
    else:
        k = 10.0 ** rng.uniform(-2.0, 2.0, m.n)
        kl, ku = k[a.lowerAddr], k[a.upperAddr]
        upper = -2.0 * kl * ku / (kl + ku)
    diag = _diag_of(m, upper, upper)
    diag[0] *= 2.0
    b = rng.standard_normal(m.n)
    b -= b.mean()
    return diag, upper, b


def _momentum_system(m, nrhs, seed):
    """First-order upwind convection-diffusion: eight random Fourier modes
    of velocity, D = 0.05 per face, diagonal = sum |off-diagonals| + 0.01."""
    rng = np.random.default_rng(seed)
    a = m.addr
    ks = rng.integers(-3, 4, size=(8, 3)).astype(np.float64)
    phases = rng.uniform(0.0, 2.0 * np.pi, 8)
    amps = rng.standard_normal((8, 3))
    amps /= np.linalg.norm(amps, axis=1, keepdims=True)
    nx, ny, nz = m.dims
    c = a.lowerAddr
    x = [(c % nx + 0.5) / nx, (c // nx % ny + 0.5) / ny, (c // (nx * ny) + 0.5) / nz]
    for d, size in enumerate(m.dims):
        x[d] = x[d] + np.where(m.axis == d, 0.5 / size, 0.0)
    flux = np.zeros(m.nf)
    for q in range(8):
        wave = np.cos(2.0 * np.pi * (ks[q, 0] * x[0] + ks[q, 1] * x[1] + ks[q, 2] * x[2])
                      + phases[q])
        flux += wave * amps[q][m.axis]
    lower = -(0.05 + np.maximum(flux, 0.0))
    upper = -(0.05 + np.maximum(-flux, 0.0))
    # the sum of the off-diagonals of every row: upper in the owner's row,
    # lower in the neighbour's
    diag = _diag_of(m, upper, lower) + 0.01
    b = rng.uniform(-1.0, 1.0, m.n) if nrhs == 1 else rng.standard_normal((nrhs, m.n))
    return diag, upper, lower, b


def _spmv_system(m, symmetric, seed):
    diag, upper, b = _pressure_system(m, "varcoeff", seed)
    rng = np.random.default_rng(seed + 1)
    lower = None if symmetric else (upper * rng.uniform(0.5, 1.5, m.nf)).astype(np.float32)
    x = rng.standard_normal(m.n).astype(np.float32)
    w = rng.uniform(0.5, 1.5, m.n).astype(np.float32) * np.sign(x)
    return diag.astype(np.float32), upper.astype(np.float32), lower, x, w.astype(np.float32)


def _dev(*arrays):
    return [None if v is None else torch.from_numpy(np.ascontiguousarray(v)).to(DEV)
            for v in arrays]


def _grid(case, kind=None):
    return _mesh(kind or case.get("mesh", "grid"), case["nx"], case["ny"], case["nz"],
                 bool(case.get("permute", False)))


# ----------------------------------------------------------------- the cases


class _State:
    pass


def _context(m, stream):
    ctx = _lib.Context(0)
    ctx.set_stream(stream.cuda_stream)
    ctx.set_topology(m.n, m.nf, *m.addr.arrays())
    return ctx


def _controls(case):
    if case["kind"] == "momentum":
        return {"solver": "cudaPBiCGStab", "tolerance": case["tol"], "maxIter": 5000}
    return {"solver": "cudaPCG", "tolerance": 1e-6, "maxIter": 5000,
            "cuda": {"chebyshevOrder": case["order"], "preconditioner": case["precond"]}}


def prepare(case, seed):
    s = _State()
    s.case, s.kind = case, case["kind"]
    if s.kind == "spmv":
        s.m = _grid(case)
        s.addr = _dev(*s.m.addr.arrays())
        s.diag, s.upper, s.lower, s.x, s.w = _dev(*_spmv_system(s.m, case["symmetric"], seed))
        s.y = torch.empty_like(s.x)
        s.dot = torch.empty(1, dtype=torch.float64, device=DEV)
        torch.cuda.synchronize()
        return s
    s.stream = torch.cuda.Stream()
    if s.kind == "batch":
        s.batch = _lib.Batch(0)
        s.batch.set_stream(s.stream.cuda_stream)
        s.sys = []
        for k, (nx, ny, nz) in enumerate(_batch_dims(case)):
            m = _mesh("grid", nx, ny, nz, False)
            s.batch.add_system(m.addr)
            s.sys.append(_dev(*_pressure_system(m, "varcoeff", 1000 * seed + k)))
        s.batch.finalize()
        s.options = _lib.default_options(**OPTIONS["batch"])
        torch.cuda.synchronize()
        return s
    s.m = _grid(case)
    if s.kind == "momentum":
        diag, upper, lower, b = _momentum_system(s.m, case["nrhs"], seed)
        opts = dict(OPTIONS["momentum"], tolerance=case["tol"])
    else:
        diag, upper, b = _pressure_system(s.m, case.get("coeffs", "varcoeff"), seed)
        lower = None
        opts = dict(OPTIONS[s.kind])
        if s.kind == "pressure":
            opts.update(chebyshevOrder=case["order"], preconditioner=case["precond"])
    if case.get("host"):
        matrix = lduMatrix(s.m.ldu, diag, upper, lower)
        s.solver = lduMatrix.solver.New("U" if lower is not None else "p", matrix, _controls(case))
        s.b = b
        return s
    s.ctx = _context(s.m, s.stream)
    s.diag, s.upper, s.lower, s.b = _dev(diag, upper, lower, b)
    s.options = _lib.default_options(**opts)
    if s.kind == "adjoint":
        s.target, = _dev(np.random.default_rng(seed + 1).standard_normal(s.m.n))
    torch.cuda.synchronize()
    return s


def run(s):
    case = s.case
    if s.kind == "spmv":
        _lib.check(_lib.load().cf_ldu_spmv_dot_noalloc(
            s.m.n, _lib.ptr(s.diag), _lib.ptr(s.upper), _lib.ptr(s.lower),
            *(_lib.ptr(a) for a in s.addr), _lib.ptr(s.x), _lib.ptr(s.w), _lib.ptr(s.y),
            _lib.ptr(s.dot), torch.cuda.current_stream().cuda_stream))
        return {"y": s.y, "dot": s.dot}
    if case.get("host"):
        psi = np.zeros_like(s.b)
        if psi.ndim == 2:
            s.solver.solveSegregated(psi, s.b)
        else:
            s.solver.solve(psi, s.b)
        return {"psi": psi}
    with torch.cuda.stream(s.stream):
        if s.kind == "batch":
            psis = [torch.zeros_like(b) for _, _, b in s.sys]
            for k, (diag, upper, _) in enumerate(s.sys):
                s.batch.set_coeffs_device(k, diag, upper)
            s.batch.solve_device(psis, [b for _, _, b in s.sys], s.options)
            return {"psi": psis}
        psi = torch.zeros_like(s.b)
        s.ctx.set_coeffs_device(s.diag, s.upper, s.lower)
        if s.kind == "momentum":
            if case["nrhs"] > 1:
                s.ctx.solve_multi_device(_lib.CF_SOLVER_PBICGSTAB, psi, s.b, s.options)
            else:
                s.ctx.solve_device(_lib.CF_SOLVER_PBICGSTAB, psi, s.b, s.options)
            return {"psi": psi}
        s.ctx.solve_device(_lib.CF_SOLVER_PCG, psi, s.b, s.options)
        if s.kind == "pressure":
            return {"psi": psi}
        g = psi - s.target
        lam, d_diag = torch.empty_like(psi), torch.empty_like(psi)
        d_upper, d_lower = torch.empty_like(s.upper), torch.empty_like(s.upper)
        perf = _lib.Performance()
        _lib.check(_lib.load().cf_solve_adjoint_device(
            s.ctx.h, _lib.CF_SOLVER_PCG, _lib.ptr(psi), _lib.ptr(g), _lib.ptr(lam),
            _lib.ptr(d_upper), _lib.ptr(d_lower), _lib.ptr(d_diag), s.options, perf))
        return {"x": psi, "db": lam, "ddiag": d_diag, "dupper": d_upper, "dlower": d_lower}


def work(case):
    """Bytes and operations one pass cannot do without: the FP64
    coefficients, source and solution once, and the addressing once."""
    if case["kind"] == "batch":
        sizes = [(nx * ny * nz, 3 * nx * ny * nz - nx * ny - ny * nz - nx * nz if nz > 1
                  else 2 * nx * ny - nx - ny) for nx, ny, nz in _batch_dims(case)]
        n, nf = sum(a for a, _ in sizes), sum(b for _, b in sizes)
    else:
        m = _grid(case)
        n, nf = m.n, m.nf
    addressing = 4 * (3 * nf + 2 * (n + 1))
    if case["kind"] == "spmv":
        faces = nf if case["symmetric"] else 2 * nf
        return {"bytes": 4 * (4 * n + faces) + addressing + 8, "flops": 2 * (n + 2 * nf) + 2 * n}
    nrhs = case.get("nrhs", 1)
    faces = 2 * nf if case["kind"] in ("momentum", "adjoint") else nf
    extra = 8 * (3 * n + 2 * nf) if case["kind"] == "adjoint" else 0
    return {"bytes": 8 * (n + faces + 2 * nrhs * n) + addressing + extra,
            "flops": 2 * nrhs * (n + 2 * nf)}


# ------------------------------------------------------------- 64-bit values


def _csr(m, diag, upper, lower):
    a = m.addr
    rows = torch.from_numpy(np.concatenate([np.arange(m.n, dtype=np.int64), a.lowerAddr,
                                            a.upperAddr])).to(DEV)
    cols = torch.from_numpy(np.concatenate([np.arange(m.n, dtype=np.int64), a.upperAddr,
                                            a.lowerAddr])).to(DEV)
    vals = torch.from_numpy(np.concatenate([diag, upper, upper if lower is None else lower]))
    return torch.sparse_coo_tensor(torch.stack([rows, cols]), vals.to(DEV),
                                   (m.n, m.n)).coalesce().to_sparse_csr()


def _cg64(A, d, b, tol=1e-13, maxiter=20000):
    """Jacobi-preconditioned CG in 64 bits, restarted on the true residual."""
    x = torch.zeros_like(b)
    limit = tol * torch.linalg.vector_norm(b)
    for _ in range(3):
        r = b - A @ x
        if torch.linalg.vector_norm(r) <= limit:
            break
        z = r / d
        p = z.clone()
        rz = r @ z
        for k in range(maxiter):
            q = A @ p
            alpha = rz / (p @ q)
            x += alpha * p
            r -= alpha * q
            if k % 50 == 49 and torch.linalg.vector_norm(r) <= limit:
                break
            z = r / d
            new = r @ z
            p = z + (new / rz) * p
            rz = new
    return x


def _bicgstab64(A, d, b, tol=1e-13, maxiter=20000):
    x = torch.zeros_like(b)
    limit = tol * torch.linalg.vector_norm(b)
    for _ in range(4):
        r = b - A @ x
        if torch.linalg.vector_norm(r) <= limit:
            break
        r0 = r.clone()
        p = r.clone()
        rho = r0 @ r
        for _ in range(maxiter):
            y = p / d
            v = A @ y
            alpha = rho / (r0 @ v)
            s = r - alpha * v
            z = s / d
            t = A @ z
            omega = (t @ s) / (t @ t)
            step = alpha * y + omega * z
            nr = s - omega * t
            if not bool(torch.isfinite(step).all()):
                break
            x += step
            r = nr
            if torch.linalg.vector_norm(r) <= limit:
                break
            new = r0 @ r
            p = r + (new / rho) * (alpha / omega) * (p - omega * v)
            rho = new
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "spmv":
        m = _grid(case)
        diag, upper, lower, x, w = _spmv_system(m, case["symmetric"], seed)
        a = m.addr
        d, u, xx, ww = (v.astype(np.float64) for v in (diag, upper, x, w))
        lo = u if lower is None else lower.astype(np.float64)
        y = (d * xx + np.bincount(a.lowerAddr, weights=u * xx[a.upperAddr], minlength=m.n)
             + np.bincount(a.upperAddr, weights=lo * xx[a.lowerAddr], minlength=m.n))
        return {"y": y, "dot": np.array([ww @ y])}
    if kind == "batch":
        out = []
        for k, (nx, ny, nz) in enumerate(_batch_dims(case)):
            m = _mesh("grid", nx, ny, nz, False)
            diag, upper, b = _pressure_system(m, "varcoeff", 1000 * seed + k)
            d, bb = _dev(diag, b)
            out.append(_cg64(_csr(m, diag, upper, None), d, bb))
        return {"psi": out}
    m = _grid(case)
    if kind == "momentum":
        diag, upper, lower, b = _momentum_system(m, case["nrhs"], seed)
        A = _csr(m, diag, upper, lower)
        d, bb = _dev(diag, b)
        if case["nrhs"] > 1:
            return {"psi": torch.stack([_bicgstab64(A, d, v) for v in bb])}
        return {"psi": _bicgstab64(A, d, bb)}
    diag, upper, b = _pressure_system(m, case.get("coeffs", "varcoeff"), seed)
    A = _csr(m, diag, upper, None)
    d, bb = _dev(diag, b)
    x = _cg64(A, d, bb)
    if kind == "pressure":
        return {"psi": x}
    target, lo, up = _dev(np.random.default_rng(seed + 1).standard_normal(m.n),
                          m.addr.lowerAddr.astype(np.int64), m.addr.upperAddr.astype(np.int64))
    lam = _cg64(A, d, x - target)
    return {"x": x, "db": lam, "ddiag": -lam * x, "dupper": -lam[lo] * x[up],
            "dlower": -lam[up] * x[lo]}
