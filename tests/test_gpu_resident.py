"""Resident inner PCG: the mesh split over the CTAs of one cluster (small
meshes) or over the SMs (128 cells per SM up to what the SMs hold), one
launch per inner solve.  Every row is formed with the graph loop's operations in the graph loop's order and
the scalars are rounded to FP32 before they are used, so the correction is
the graph loop's (clusterMaxCells < 0) bit for bit although the FP64 sums fold
in another order.  The sizes sit at the edges: the smallest mesh that is
split, the first that needs another row per thread, the ones that leave
registers for shared memory, and the first too large."""
import threading

import numpy as np
import pytest

from metal4foam_b200 import _lib, mesh

pytestmark = pytest.mark.gpu

FIELDS = ("initialResidual", "finalResidual", "nIterations", "nRestarts", "converged", "singular",
          "stagnated", "deflated", "polished", "normFactor", "residualL2", "chebBeta")


def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def context(s):
    ctx = _lib.Context(0)
    ctx.set_topology(s.addr.n, s.addr.nf, *s.addr.arrays())
    ctx.set_coeffs(s.diag, s.upper, None)
    return ctx


def solve(ctx, s, cluster=0, **kw):
    x = s.psi.copy()
    l0 = ctx.kernel_launches()
    p = ctx.solve(_lib.CF_SOLVER_PCG, x, s.source,
                  _lib.default_options(clusterMaxCells=cluster, **kw))
    return x, p, ctx.kernel_launches() - l0


def chain_of_grids(cells, seed):
    """Two unconnected grids, one of them 2 x 3 cells across."""
    a = mesh.structured_faces((2, 3, cells // 12))
    b = mesh.structured_faces((30, cells // 60))
    na, nb = 6 * (cells // 12), 30 * (cells // 60)
    low = np.concatenate([a[0], b[0] + na])
    upp = np.concatenate([a[1], b[1] + na])
    n = na + nb
    rng = np.random.default_rng(seed)
    addr = mesh.ldu_addressing(n, low, upp)
    upper = -rng.uniform(0.5, 2.0, addr.nf)
    diag = 0.01 - (np.bincount(low, upper, n) + np.bincount(upp, upper, n))
    return mesh.LduSystem("chain", addr, diag, upper, None, rng.standard_normal(n), np.zeros(n))


def random_graph(n, seed):
    """At most six random neighbours per cell: no locality to find."""
    rng = np.random.default_rng(seed)
    pairs = np.concatenate([np.stack([np.arange(n), rng.permutation(n)], 1) for _ in range(3)])
    pairs = pairs[pairs[:, 0] != pairs[:, 1]]
    key = np.unique(np.minimum(pairs[:, 0], pairs[:, 1]) * n + np.maximum(pairs[:, 0], pairs[:, 1]))
    low, upp = (key // n).astype(np.int32), (key % n).astype(np.int32)
    addr = mesh.ldu_addressing(n, low, upp)
    upper = -rng.uniform(0.5, 2.0, addr.nf)
    diag = 0.05 - (np.bincount(low, upper, n) + np.bincount(upp, upper, n))
    return mesh.LduSystem("random", addr, diag, upper, None, rng.standard_normal(n), np.zeros(n))


CASES = {
    "first_size": (lambda m: mesh.poisson2d(128, m, seed=1), {}),
    "one_row_each": (lambda m: mesh.varcoeff3d((16, 16, m), seed=2, permute=True), {}),
    "two_rows": (lambda m: mesh.varcoeff3d((16, 16, m + 1), seed=3), dict(deflate="off")),
    "prism_rcm": (lambda m: mesh.prism3d((41, 37, 29), seed=4), dict(tolerance=1e-9)),
    "jacobi": (lambda m: mesh.poisson2d(211, 307, seed=5),
               dict(chebyshevOrder=1, maxIter=3000)),
    "order2_ips3": (lambda m: mesh.varcoeff3d((37, 35, 33), seed=6, permute=True),
                    dict(chebyshevOrder=2, iterationsPerSync=3)),
    "max_iter": (lambda m: mesh.varcoeff3d((41, 40, 39), seed=7, permute=True),
                 dict(maxIter=17, maxRestarts=2)),
    "unconnected": (lambda m: chain_of_grids(150 * m, 8), {}),
    "random_graph": (lambda m: random_graph(140 * m, 9), {}),
    "rows_10": (lambda m: mesh.poisson2d(16 * m, 160, seed=10), dict(chebyshevOrder=4)),
    "shared_rows": (lambda m: mesh.varcoeff3d((16 * m // 10, 20, 81), seed=11), {}),
    "last_size": (lambda m: mesh.varcoeff3d((m, 64, 88), seed=12), dict(maxIter=60)),
}


@pytest.mark.parametrize("name", CASES)
def test_resident_equals_graph(require_gpu, name):
    make, kw = CASES[name]
    s = make(sms())
    ctx = context(s)
    xg, pg, lg = solve(ctx, s, -1, **kw)
    # the split is made by the third solve on a topology
    _, p2, l2 = solve(ctx, s, **kw)
    assert l2 == lg and p2.nIterations == pg.nIterations
    xr, pr, lr = solve(ctx, s, **kw)
    assert lr < lg and lr <= 10 * (pr.nRestarts + 2), (lr, lg)     # one launch per inner solve
    for f in FIELDS:
        assert getattr(pr, f) == getattr(pg, f), (f, getattr(pr, f), getattr(pg, f))
    assert np.array_equal(xr, xg)
    # (another 1e-12: the FP64 sum of n FP32 magnitudes in another order)
    assert pr.finalResSum32 == pytest.approx(pg.finalResSum32, rel=1e-12)
    ctx.close()


def chain_1d(n, seed):
    low = np.arange(n - 1, dtype=np.int32)
    addr = mesh.ldu_addressing(n, low, low + 1)
    rng = np.random.default_rng(seed)
    upper = -rng.uniform(0.5, 2.0, n - 1)
    diag = 0.1 - (np.bincount(low, upper, n) + np.bincount(low + 1, upper, n))
    return mesh.LduSystem("chain", addr, diag, upper, None, rng.standard_normal(n), np.zeros(n))


# one cluster: one CTA, its last row, a second CTA, every number of rows per
# thread, no faces at all, the largest meshes of each width
CLUSTER = {
    "one_cell": (lambda: chain_1d(1, 1), {}),
    "one_cta": (lambda: mesh.poisson2d(16, 16, seed=2), {}),
    "two_ctas": (lambda: chain_1d(257, 3), dict(chebyshevOrder=3)),
    "sixteen_ctas": (lambda: mesh.poisson2d(63, 65, seed=4), dict(deflate="off", tolerance=1e-7)),
    "two_rows": (lambda: mesh.varcoeff3d((100, 71), seed=5, permute=False), {}),
    "three_rows_3d": (lambda: mesh.varcoeff3d((25, 23, 21), seed=6, permute=False),
                      dict(iterationsPerSync=4)),
    "four_rows": (lambda: mesh.poisson2d(128, 128, seed=7), dict(chebyshevOrder=4)),
    "jacobi": (lambda: mesh.poisson2d(90, 80, seed=8), dict(chebyshevOrder=1, maxIter=3000)),
    "max_iter": (lambda: mesh.varcoeff3d((80, 50), seed=9, permute=False),
                 dict(maxIter=23, maxRestarts=3)),
    "no_faces": (lambda: mesh.LduSystem("diag", mesh.ldu_addressing(
        900, np.zeros(0, np.int32), np.zeros(0, np.int32)), np.linspace(1.0, 2.0, 900),
        np.zeros(0), None, np.linspace(-1.0, 1.0, 900), np.zeros(900)), {}),
    "six_rows_3d": (lambda: mesh.varcoeff3d((31, 29, 27), seed=10, permute=True), {}),
    "last_3d": (lambda: mesh.varcoeff3d((30, 35, 26), seed=11), {}),
    "last_prism": (lambda: mesh.prism3d((32, 32, 16), seed=12), {}),
    "ten_rows_2d": (lambda: mesh.poisson2d(256, 160, seed=13), {}),
}


@pytest.mark.parametrize("name", CLUSTER)
def test_cluster_equals_graph(require_gpu, name):
    make, kw = CLUSTER[name]
    s = make()
    ctx = context(s)
    for _ in range(1 if s.n <= 16384 else 2):
        xg, pg, lg = solve(ctx, s, -1, **kw)
    for _ in range(2):
        xr, pr, lr = solve(ctx, s, **kw)
        assert lr < lg and lr <= 10 * (pr.nRestarts + 2), (lr, lg)
        for f in FIELDS:
            assert getattr(pr, f) == getattr(pg, f), (f, getattr(pr, f), getattr(pg, f))
        assert np.array_equal(xr, xg)
        assert pr.finalResSum32 == pytest.approx(pg.finalResSum32, rel=1e-12)
    # a wait limit of one poll: the graph loop takes over, nothing else changes
    ctx.set_wait_limit(1)
    x1, p1, _ = solve(ctx, s, **kw)
    assert np.array_equal(x1, xg) and p1.nIterations == pg.nIterations
    ctx.set_wait_limit(0)
    x2, p2, l2 = solve(ctx, s, **kw)
    assert l2 == lr and np.array_equal(x2, xg)
    ctx.close()


# cudaPBiCGStab in one cluster: one 256-row block, its last row and a second
# block, one block per CTA, two blocks per CTA, every number of blocks per
# thread, the largest mesh
BICG = {
    "one_block": (lambda: mesh.upwind3d((16, 15), seed=1), {}),
    "two_blocks": (lambda: mesh.upwind3d((257, 1, 1), seed=2), {}),
    "sixteen_ctas": (lambda: mesh.upwind3d((64, 64), seed=3), dict(tolerance=1e-6)),
    "nine_ctas": (lambda: mesh.upwind3d((17, 241, 1), seed=4), {}),
    "three_blocks": (lambda: mesh.upwind3d((25, 23, 21), seed=5), {}),
    "six_blocks": (lambda: mesh.upwind3d((30, 29, 25), seed=6), dict(iterationsPerSync=1)),
    "max_iter": (lambda: mesh.upwind3d((25, 23, 21), seed=7), dict(maxIter=9, maxRestarts=2)),
    "symmetric": (lambda: mesh.varcoeff3d((20, 18, 16), seed=8), {}),
    "prism": (lambda: mesh.prism3d((24, 24, 16), seed=9), dict(tolerance=1e-6)),
    "ten_blocks": (lambda: mesh.upwind3d((32, 32, 40), seed=10), dict(tolerance=1e-6)),
}


def one_cell_more(s):
    """s with a cell hung on its last one."""
    low, upp = (np.append(a, v).astype(np.int32) for a, v in zip(s.addr.arrays()[:2], (s.n - 1, s.n)))
    addr = mesh.ldu_addressing(s.n + 1, low, upp)
    return mesh.LduSystem("more", addr, np.append(s.diag, 2.0), np.append(s.upper, -0.5),
                          np.append(s.lower, -1.0), np.append(s.source, 1.0), np.zeros(s.n + 1))


# one CTA per SM (1 m groups of 256 rows fill the m SMs once): the first
# mesh too large for the cluster, a group of one row, the last and the first
# number of groups before the blocks of each sum wrap (5, 6 and 8 per SM) for
# each row width, numbers of groups per CTA that no kernel has, the largest
# mesh and the first too large (launches as the graph loop)
BICG_SMS = {
    "first": (lambda m: mesh.upwind3d((37, 36, 31), seed=11), {}),
    "one_row_more_2d": (lambda m: one_cell_more(mesh.upwind3d((2 * m, 256), seed=12)),
                        dict(maxIter=40)),
    "prism_5": (lambda m: mesh.prism3d((m // 2, 32, 64), seed=13), dict(maxIter=60)),
    "prism_7": (lambda m: mesh.prism3d((m // 2, 52, 64), seed=14), dict(maxIter=60)),
    "ab_full_3d": (lambda m: mesh.upwind3d((m, 32, 48), seed=15), {}),
    "ab_wraps_3d": (lambda m: mesh.upwind3d((m, 32, 49), seed=16), dict(iterationsPerSync=3)),
    "cd_full_2d": (lambda m: mesh.upwind3d((m, 1280), seed=17), dict(maxIter=60)),
    "cd_wraps_2d": (lambda m: mesh.upwind3d((m, 1291), seed=18), dict(maxIter=60)),
    "e_wraps_2d": (lambda m: mesh.upwind3d((m, 2051), seed=19), dict(maxIter=40)),
    "symmetric_9": (lambda m: mesh.varcoeff3d((m, 45, 50), seed=20), dict(maxIter=50)),
    "last": (lambda m: mesh.upwind3d((m, 64, 96), seed=21), dict(maxIter=30)),
    "too_large": (lambda m: mesh.upwind3d((m, 64, 97), seed=22), dict(maxIter=30)),
}


@pytest.mark.parametrize("name", [*BICG, *BICG_SMS])
def test_bicgstab_equals_graph(require_gpu, name):
    """Every sum folds in the graph loop's order, so every field is equal."""
    if name in BICG:
        make, kw = BICG[name]
        s = make()
    else:
        make, kw = BICG_SMS[name]
        s = make(sms())
    ctx = _lib.Context(0)
    ctx.set_topology(s.addr.n, s.addr.nf, *s.addr.arrays())
    ctx.set_coeffs(s.diag, s.upper, s.lower)

    def run(cluster):
        x = np.zeros(s.n)
        l0 = ctx.kernel_launches()
        opts = dict(tolerance=1e-8, maxIter=5000, clusterMaxCells=cluster)
        opts.update(kw)
        p = ctx.solve(_lib.CF_SOLVER_PBICGSTAB, x, s.source, _lib.default_options(**opts))
        return x, p, ctx.kernel_launches() - l0

    xg, pg, lg = run(-1)
    for _ in range(2):
        xr, pr, lr = run(0)
        assert (lr == lg) if name == "too_large" else (lr < lg), (lr, lg)
        for f in FIELDS + ("finalResSum32",):
            assert getattr(pr, f) == getattr(pg, f), (f, getattr(pr, f), getattr(pg, f))
        assert np.array_equal(xr, xg)
    ctx.set_wait_limit(1)
    x1, p1, _ = run(0)
    assert np.array_equal(x1, xg) and p1.nIterations == pg.nIterations
    ctx.set_wait_limit(0)
    # three components, each in a cluster of its own on the shared split or in
    # turn on all SMs
    rng = np.random.default_rng(12)
    b = rng.standard_normal((3, s.n))
    limit = kw.get("maxIter", 5000)
    opts = _lib.default_options(tolerance=1e-7, maxIter=limit)
    psi = np.zeros((3, s.n))
    perfs = ctx.solve_multi(_lib.CF_SOLVER_PBICGSTAB, psi, b, opts)
    for k in range(3):
        x = np.zeros(s.n)
        p = ctx.solve(_lib.CF_SOLVER_PBICGSTAB, x, b[k],
                      _lib.default_options(tolerance=1e-7, maxIter=limit, clusterMaxCells=-1))
        assert np.array_equal(psi[k], x) and p.nIterations == perfs[k].nIterations
    ctx.close()


def test_resident_size_limits(require_gpu):
    """Just below the first size and just above the last: the graph loop
    (same launches with and without)."""
    m = sms()
    for s in (mesh.varcoeff3d((128, m - 1), seed=1, permute=False),
              mesh.varcoeff3d((m, 64, 97), seed=2, permute=False)):
        ctx = context(s)
        for _ in range(2):
            _, pg, lg = solve(ctx, s, -1, maxIter=40)
        _, pr, lr = solve(ctx, s, maxIter=40)
        assert lr == lg and pr.nIterations == pg.nIterations
        ctx.close()


def test_resident_inner_entry_new_coeffs_and_transpose(require_gpu):
    """cf_pcg runs through it too; new coefficients, a staged transpose and a
    new topology on the same context are picked up."""
    s = mesh.varcoeff3d((40, 30, 20), seed=13, permute=True)
    ctx = context(s)
    for _ in range(3):
        st = ctx.pcg(s.source, 1e-3 * np.abs(s.source).sum(), 200, chebOrder=8, chebBeta=2.0)
    d0 = ctx.delta(s.n)
    assert st.converged
    ctx.set_spmv_config(blockSize=128)            # the graph loop in another launch shape
    st1 = ctx.pcg(s.source, 1e-3 * np.abs(s.source).sum(), 200, chebOrder=8, chebBeta=2.0)
    assert abs(st1.nIterations - st.nIterations) <= 1
    assert np.linalg.norm(ctx.delta(s.n) - d0) <= 1e-3 * np.linalg.norm(d0)
    ctx.set_spmv_config()
    s2 = mesh.varcoeff3d((40, 30, 20), seed=14, permute=True)
    ctx.set_topology(s2.addr.n, s2.addr.nf, *s2.addr.arrays())
    ctx.set_coeffs(s2.diag, s2.upper, None)
    solve(ctx, s2, -1)
    for scale in (1.0, 3.0):
        ctx.set_coeffs(scale * s2.diag, scale * s2.upper, None)
        for on in (False, True):
            ctx.set_transpose(on)
            xg, pg, _ = solve(ctx, s2, -1)
            xr, pr, _ = solve(ctx, s2)
            assert np.array_equal(xr, xg) and pr.nIterations == pg.nIterations
        ctx.set_transpose(False)
    ctx.close()


def test_resident_wait_runs_out(require_gpu):
    """With a wait limit of one poll a CTA gives up on its neighbours: the
    launch ends and the inner solve runs through the graph loop instead."""
    s = mesh.varcoeff3d((40, 40, 40), seed=15, permute=True)
    ctx = context(s)
    for _ in range(2):
        xg, pg, lg = solve(ctx, s, -1)
    ctx.set_wait_limit(1)
    x1, p1, l1 = solve(ctx, s)
    assert l1 > lg and np.array_equal(x1, xg) and p1.nIterations == pg.nIterations
    ctx.set_wait_limit(0)
    xr, pr, lr = solve(ctx, s)
    assert lr < lg and np.array_equal(xr, xg) and pr.nIterations == pg.nIterations
    ctx.close()


def test_resident_from_two_threads(require_gpu):
    """One resident launch at a time per device: solves on other threads take
    the graph loop meanwhile, with the same result."""
    ss = [mesh.varcoeff3d((40, 40, 20 + k), seed=20 + k, permute=True) for k in range(3)]
    ctxs = [context(s) for s in ss]
    for _ in range(2):
        ref = [solve(c, s, -1) for c, s in zip(ctxs, ss)]
    out = [[] for _ in ss]

    def work(k):
        for _ in range(5):
            out[k].append(solve(ctxs[k], ss[k]))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(ss))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(len(ss)):
        assert len(out[k]) == 5
        for x, p, _ in out[k]:
            assert np.array_equal(x, ref[k][0]) and p.nIterations == ref[k][1].nIterations
        ctxs[k].close()


def test_bicgstab_with_the_other_column_stream(require_gpu):
    """A switch to 32-bit columns (and back) after a resident solve: the
    graph loop on that stream, alone and for several components."""
    s = mesh.upwind3d((40, 36, 31), seed=30)
    ctx = _lib.Context(0)
    ctx.set_topology(s.addr.n, s.addr.nf, *s.addr.arrays())
    ctx.set_coeffs(s.diag, s.upper, s.lower)
    b = np.random.default_rng(31).standard_normal((2, s.n))
    launches = {}
    for bits in (16, 32, 16):
        ctx.set_spmv_config(indexBits=bits)
        out = []
        for cluster in (-1, 0):
            x = np.zeros(s.n)
            l0 = ctx.kernel_launches()
            opts = _lib.default_options(tolerance=1e-8, maxIter=2000, clusterMaxCells=cluster)
            p = ctx.solve(_lib.CF_SOLVER_PBICGSTAB, x, s.source, opts)
            launches[bits, cluster] = ctx.kernel_launches() - l0
            psi = np.zeros((2, s.n))
            q = ctx.solve_multi(_lib.CF_SOLVER_PBICGSTAB, psi, b, opts)
            assert p.converged and all(r.converged for r in q)
            out.append((x, psi, p.nIterations, [r.nIterations for r in q]))
        assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
        assert out[0][2:] == out[1][2:]
    assert launches[16, 0] < launches[16, -1] and launches[32, 0] == launches[32, -1]
    ctx.close()


def test_bicgstab_components_on_several_threads(require_gpu):
    """Two multi-RHS solves and a cudaPCG solve at once: their launches take
    turns on the SMs, every result is the one of the graph loop."""
    ms = [mesh.upwind3d((40, 36, 31), seed=32), mesh.upwind3d((48, 45, 40), seed=33)]
    sp = mesh.varcoeff3d((40, 40, 22), seed=34, permute=True)
    ctxs = []
    for s in ms:
        ctx = _lib.Context(0)
        ctx.set_topology(s.addr.n, s.addr.nf, *s.addr.arrays())
        ctx.set_coeffs(s.diag, s.upper, s.lower)
        ctxs.append(ctx)
    cp = context(sp)
    b = [np.random.default_rng(35 + k).standard_normal((3, s.n)) for k, s in enumerate(ms)]

    def multi(k, cluster):
        psi = np.zeros((3, ms[k].n))
        p = ctxs[k].solve_multi(_lib.CF_SOLVER_PBICGSTAB, psi, b[k], _lib.default_options(
            tolerance=1e-8, maxIter=2000, clusterMaxCells=cluster))
        return psi, [q.nIterations for q in p]

    ref = [multi(k, -1) for k in range(2)]
    for _ in range(2):
        refp = solve(cp, sp, -1)
    out = [[], [], []]

    def work(k):
        for _ in range(4):
            out[k].append(multi(k, 0) if k < 2 else solve(cp, sp))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        assert len(out[k]) == 4
        for psi, its in out[k]:
            assert np.array_equal(psi, ref[k][0]) and its == ref[k][1]
        ctxs[k].close()
    assert len(out[2]) == 4 and all(np.array_equal(x, refp[0]) for x, _, _ in out[2])
    cp.close()
