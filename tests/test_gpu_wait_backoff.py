"""After the waits of a whole inner solve have run out, the following inner
solves go through the graph loop, for longer every time; a call of
set_wait_limit or a new topology tries at once again.  Waits are made to run
out by a limit of one poll, attempts are counted by the extra launch."""
import numpy as np
import pytest

from metal4foam_b200 import _lib, mesh

pytestmark = pytest.mark.gpu

PCG, BICG = _lib.CF_SOLVER_PCG, _lib.CF_SOLVER_PBICGSTAB
SOLVES = 24


def run(ctx, s, solver, cluster=0):
    x = np.zeros(s.n)
    l0 = ctx.kernel_launches()
    ctx.solve(solver, x, s.source,
              _lib.default_options(clusterMaxCells=cluster, maxIter=30, maxRestarts=0))
    return x, ctx.kernel_launches() - l0


@pytest.mark.parametrize("make,solver", [
    (lambda: mesh.poisson2d(90, 80, seed=1), PCG),
    (lambda: mesh.poisson2d(160, 150, seed=2), PCG),
    (lambda: mesh.varcoeff3d((44, 42, 40), seed=3, permute=True), PCG),
    (lambda: mesh.upwind3d((24, 23, 22), seed=4), BICG),
    (lambda: mesh.upwind3d((40, 38, 36), seed=5), BICG),
], ids=["cluster", "cluster_third", "sms", "bicg_cluster", "bicg_sms"])
def test_attempts_become_rare(require_gpu, make, solver):
    s = make()
    ctx = _lib.Context(0)

    small = mesh.ldu_addressing(2, np.zeros(1, np.int32), np.ones(1, np.int32))

    def topology():
        ctx.set_topology(small.n, small.nf, *small.arrays())   # (the same again is no new one)
        ctx.set_topology(s.addr.n, s.addr.nf, *s.addr.arrays())
        ctx.set_coeffs(s.diag, s.upper, s.lower)
        return [run(ctx, s, solver, -1) for _ in range(2)][1]

    xl, loop = topology()
    _, whole = run(ctx, s, solver)
    assert whole < loop
    ctx.set_wait_limit(1)
    tried = []
    for _ in range(SOLVES):                        # one inner solve each
        x, n = run(ctx, s, solver)
        assert np.array_equal(x, xl)               # (the graph loop's, as documented)
        tried.append(n - loop)
    # attempts at solve 1, 4 (2 skipped), 9 (4), 18 (8)
    expect = [int(k in (0, 3, 8, 17)) for k in range(SOLVES)]
    assert tried == expect, tried
    if solver == BICG:
        # components start where the context is (8 more solves skipped, then 16)
        b = np.stack([s.source, 2.0 * s.source, -s.source])
        opts = dict(maxIter=30, maxRestarts=0)
        psi = np.zeros((3, s.n))
        counts = []
        for cluster in (-1, 0, 0):
            l0 = ctx.kernel_launches()
            ctx.solve_multi(BICG, psi, b, _lib.default_options(clusterMaxCells=cluster, **opts))
            counts.append(ctx.kernel_launches() - l0)
        assert counts[0] == counts[1] == counts[2], counts
    ctx.set_wait_limit(0)
    assert run(ctx, s, solver)[1] == whole
    ctx.set_wait_limit(1)
    assert [run(ctx, s, solver)[1] - loop for _ in range(2)] == [1, 0]
    topology()                                     # (keeps the limit, forgets the waits)
    assert run(ctx, s, solver)[1] == loop + 1
    ctx.set_wait_limit(0)
    assert run(ctx, s, solver)[1] == whole
    ctx.close()
