"""clusterMaxCells > 0 is the largest mesh that runs in a cluster or as one
launch: one cell below the mesh's size the launches (and bits) are those of
clusterMaxCells < 0, at its size those of the default."""
import numpy as np
import pytest

from metal4foam_b200 import _lib, mesh

pytestmark = pytest.mark.gpu

PCG, BICG = _lib.CF_SOLVER_PCG, _lib.CF_SOLVER_PBICGSTAB


def run(ctx, s, solver, limit, **kw):
    x = np.zeros(s.n)
    l0 = ctx.kernel_launches()
    ctx.solve(solver, x, s.source, _lib.default_options(clusterMaxCells=limit, **kw))
    return x, ctx.kernel_launches() - l0


@pytest.mark.parametrize("make,solver,kw", [
    (lambda: mesh.poisson2d(80, 70, seed=1), PCG, {}),
    (lambda: mesh.poisson2d(160, 150, seed=2), PCG, {}),
    (lambda: mesh.varcoeff3d((44, 42, 40), seed=3, permute=True), PCG, {}),
    (lambda: mesh.upwind3d((20, 19, 18), seed=4), BICG, {}),
    (lambda: mesh.upwind3d((40, 38, 36), seed=5), BICG, {}),
    # rows of eight neighbours: the cluster kernel for those
    (lambda: wide(60, 50, 6), PCG, {}),
], ids=["cluster", "cluster_third", "sms", "bicg_cluster", "bicg_sms", "wide_rows"])
def test_limit(require_gpu, make, solver, kw):
    s = make()
    ctx = _lib.Context(0)
    ctx.set_topology(s.addr.n, s.addr.nf, *s.addr.arrays())
    ctx.set_coeffs(s.diag, s.upper, s.lower)
    for _ in range(2):
        xl, loop = run(ctx, s, solver, -1, **kw)
    xd, default = run(ctx, s, solver, 0, **kw)
    assert default < loop
    for limit, x, launches in ((s.n - 1, xl, loop), (s.n, xd, default), (1, xl, loop)):
        y, got = run(ctx, s, solver, limit, **kw)
        assert got == launches and np.array_equal(y, x), limit
    if solver == BICG:
        b = np.stack([s.source, 2.0 * s.source, -s.source])
        counts = []
        for limit in (-1, s.n - 1, s.n, 0):
            psi = np.zeros((3, s.n))
            l0 = ctx.kernel_launches()
            ctx.solve_multi(BICG, psi, b, _lib.default_options(clusterMaxCells=limit))
            counts.append(ctx.kernel_launches() - l0)
        assert counts[0] == counts[1] and counts[2] == counts[3] < counts[0], counts
    ctx.close()


def wide(nx, ny, seed):
    """A 2-D grid with the diagonal neighbours."""
    i = np.arange(nx * ny).reshape(ny, nx)
    pairs = [(i[:, :-1], i[:, 1:]), (i[:-1], i[1:]), (i[:-1, :-1], i[1:, 1:]),
             (i[:-1, 1:], i[1:, :-1])]
    low = np.concatenate([a.ravel() for a, _ in pairs])
    upp = np.concatenate([b.ravel() for _, b in pairs])
    order = np.lexsort((upp, low))
    low, upp = low[order].astype(np.int32), upp[order].astype(np.int32)
    n = nx * ny
    rng = np.random.default_rng(seed)
    addr = mesh.ldu_addressing(n, low, upp)
    upper = -rng.uniform(0.5, 2.0, addr.nf)
    diag = 0.1 - (np.bincount(low, upper, n) + np.bincount(upp, upper, n))
    return mesh.LduSystem("wide", addr, diag, upper, None, rng.standard_normal(n), np.zeros(n))


def test_limit_of_a_batch(require_gpu):
    """The largest system decides."""
    # (four kernels, more launches than the batched loop counts)
    systems = [mesh.poisson2d(60, 50, seed=7), mesh.varcoeff3d((30, 28, 26), seed=8),
               mesh.prism3d((12, 11, 10), seed=9), mesh.poisson2d(30, 20, seed=10)]
    bt = _lib.Batch(0)
    for s in systems:
        bt.add_system(s.addr)
    bt.finalize("auto")
    for k, s in enumerate(systems):
        bt.set_coeffs(k, s.diag, s.upper)
    n = max(s.n for s in systems)
    counts = []
    for limit in (-1, -1, n - 1, n, 0):
        l0 = bt.kernel_launches()
        bt.solve([np.zeros(s.n) for s in systems], [s.source for s in systems],
                 _lib.default_options(clusterMaxCells=limit))
        counts.append(bt.kernel_launches() - l0)
    loop, at_limit, whole, default = counts[1:]
    assert loop == at_limit and whole == default != loop, counts
    bt.close()


def test_limit_of_gamg_levels(require_gpu):
    """The finest level of the cluster decides, not the mesh."""
    s = mesh.varcoeff3d((29, 28, 27), seed=9)
    ctx = _lib.Context(0)
    ctx.set_topology(s.addr.n, s.addr.nf, *s.addr.arrays())
    ctx.set_coeffs(s.diag, s.upper, None)
    kw = dict(preconditioner="GAMG", tolerance=1e-8)
    x0, default = run(ctx, s, PCG, 0, **kw)
    x0, default = run(ctx, s, PCG, 0, **kw)
    xl, loop = run(ctx, s, PCG, -1, **kw)
    level = max(n for n in ctx.gamg_levels()[1:] if n <= 4096)
    assert default < loop and np.array_equal(x0, xl)
    for limit, launches in ((1, loop), (level - 1, loop), (level, default), (s.n, default)):
        y, got = run(ctx, s, PCG, limit, **kw)
        assert got == launches and np.array_equal(y, x0), limit
    ctx.close()
