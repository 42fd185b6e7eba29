"""Which solves on a topology make the split of a mesh, and meshes without
locality, which keep the graph loop."""
import numpy as np
import pytest

from metal4foam_b200 import _lib, mesh

pytestmark = pytest.mark.gpu


def scattered(dims, seed):
    """An upwind mesh with its cells numbered at random."""
    s = mesh.upwind3d(dims, seed=seed)
    p = np.random.default_rng(seed).permutation(s.n)
    low, upp = s.addr.arrays()[:2]
    a, b = p[low], p[upp]
    order = np.lexsort((np.maximum(a, b), np.minimum(a, b)))
    addr = mesh.ldu_addressing(s.n, np.minimum(a, b)[order].astype(np.int32),
                               np.maximum(a, b)[order].astype(np.int32))
    upper = np.where(a > b, s.lower, s.upper)[order]
    lower = np.where(a > b, s.upper, s.lower)[order]
    diag, source = np.empty(s.n), np.empty(s.n)
    diag[p], source[p] = s.diag, s.source
    return mesh.LduSystem("scattered", addr, diag, upper, lower, source, np.zeros(s.n))


def random_links(n, seed):
    """At most six random neighbours per cell."""
    rng = np.random.default_rng(seed)
    a = np.tile(np.arange(n), 3)
    b = np.concatenate([rng.permutation(n) for _ in range(3)])
    key = np.unique(np.minimum(a, b)[a != b] * n + np.maximum(a, b)[a != b])
    low, upp = (key // n).astype(np.int32), (key % n).astype(np.int32)
    addr = mesh.ldu_addressing(n, low, upp)
    upper = -rng.uniform(0.5, 2.0, addr.nf)
    diag = 0.05 - (np.bincount(low, upper, n) + np.bincount(upp, upper, n))
    return mesh.LduSystem("links", addr, diag, upper, None, rng.standard_normal(n), np.zeros(n))


def context(s):
    ctx = _lib.Context(0)
    ctx.set_topology(s.addr.n, s.addr.nf, *s.addr.arrays())
    ctx.set_coeffs(s.diag, s.upper, s.lower)
    return ctx


def solve(ctx, s, solver, cluster=0, **kw):
    x = np.zeros(s.n)
    l0 = ctx.kernel_launches()
    ctx.solve(solver, x, s.source, _lib.default_options(clusterMaxCells=cluster, **kw))
    return x, ctx.kernel_launches() - l0


# the split is made by the first solve, unless it costs more than it gives
# there: halos of most of the mesh, many cells
@pytest.mark.parametrize("make,at_once", [
    (lambda: scattered((13, 13, 12), 2), True),
    (lambda: scattered((28, 28, 28), 3), False),
    (lambda: mesh.upwind3d((32, 32, 32), seed=4), True),
    (lambda: mesh.upwind3d((33, 32, 32), seed=5), False),
], ids=["scattered_2K", "scattered_22K", "natural_32768", "natural_33792"])
def test_first_bicgstab_solve_of_a_topology(require_gpu, make, at_once):
    s = make()
    ctx = context(s)
    x1, first = solve(ctx, s, _lib.CF_SOLVER_PBICGSTAB)
    x2, second = solve(ctx, s, _lib.CF_SOLVER_PBICGSTAB)
    xg, loop = solve(ctx, s, _lib.CF_SOLVER_PBICGSTAB, -1)
    assert (first < loop) if at_once else (first == loop), (first, loop)
    assert second < loop
    assert np.array_equal(x1, xg) and np.array_equal(x2, xg)
    ctx.close()


# cudaPCG in one cluster: the split of the larger 3-D meshes is made by the
# third solve; the kernel that runs before has one more launch per restart
@pytest.mark.parametrize("dims,at_once", [((22, 21, 17), True), ((24, 23, 21), False),
                                          ((128, 100), True)])
def test_first_pcg_solve_of_a_small_topology(require_gpu, dims, at_once):
    s = mesh.varcoeff3d(dims, seed=6, permute=False)
    ctx = context(s)
    launches = [solve(ctx, s, _lib.CF_SOLVER_PCG)[1] for _ in range(4)]
    assert launches[0] == launches[1] and launches[2] == launches[3]
    assert (launches[2] == launches[0]) if at_once else (launches[2] < launches[0]), launches
    ctx.close()


# six neighbours per cell at random: a cluster and, at the last size, the split
# over the SMs would have too many halo values
@pytest.mark.parametrize("n,whole", [(20000, True), (60000, True), (200000, False)])
def test_splits_without_locality(require_gpu, n, whole):
    s = random_links(n, n)
    ctx = context(s)
    for _ in range(2):
        xg, loop = solve(ctx, s, _lib.CF_SOLVER_PCG, -1)
    x, launches = solve(ctx, s, _lib.CF_SOLVER_PCG)
    assert (launches < loop) if whole else (launches == loop), (launches, loop)
    assert np.array_equal(x, xg)
    ctx.close()
