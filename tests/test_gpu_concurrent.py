"""Solves on several host threads: what a solve returns does not depend on
what the other threads do.

The systems have diagonal entries of both signs and a source whose z.r =
sum r^2 / d cancels to 1e-16 of its terms, so two orders of that sum give
different iterates: a solve that took another form than it takes alone would
show.  Nothing converges; three iterations are compared."""
import threading

import numpy as np
import pytest

from metal4foam_b200 import _lib, mesh

pytestmark = pytest.mark.gpu

OPTS = dict(chebyshevOrder=1, deflate="off", maxIter=3, maxRestarts=0, tolerance=1e-14)


def cancelling(dims, seed):
    low, upp = mesh.structured_faces(dims)[:2]
    n = int(np.prod(dims))
    rng = np.random.default_rng(seed)
    addr = mesh.ldu_addressing(n, low, upp)
    upper = -rng.uniform(0.1, 0.3, addr.nf)
    # powers of two: z r = r^2 / d has no rounding
    diag = rng.choice([1.0, 2.0, 4.0], n) * rng.choice([-1.0, 1.0], n)
    r = rng.standard_normal(n).astype(np.float32).astype(np.float64)
    free = rng.permutation(n)[:12]      # each cancels what is left, to FP32 accuracy
    r[free] = 0.0
    for c in free:
        t = r * r / diag
        if abs(t.sum()) < 1e-11 * np.abs(t).sum():
            break
        diag[c] = -np.sign(t.sum()) * abs(diag[c])
        r[c] = float(np.float32(np.sqrt(abs(t.sum() * diag[c]))))
    return mesh.LduSystem("cancelling", addr, diag, upper, None, r, np.zeros(n))


def context(s):
    ctx = _lib.Context(0)
    ctx.set_topology(s.addr.n, s.addr.nf, *s.addr.arrays())
    ctx.set_coeffs(s.diag, s.upper, s.lower)
    return ctx


def solve(ctx, s, cluster=0):
    x = np.zeros(s.n)
    ctx.solve(_lib.CF_SOLVER_PCG, x, s.source, _lib.default_options(clusterMaxCells=cluster, **OPTS))
    return x


def batch(systems):
    bt = _lib.Batch(0)
    for s in systems:
        bt.add_system(s.addr)
    bt.finalize("auto")
    for i, s in enumerate(systems):
        bt.set_coeffs(i, s.diag, s.upper)
    return bt


def batch_solve(bt, systems):
    xs = [np.zeros(s.n) for s in systems]
    bt.solve(xs, [s.source for s in systems], _lib.default_options(**OPTS))
    return xs


def test_results_do_not_depend_on_other_threads(require_gpu):
    """Three contexts on the split over the SMs and a batch with cooperative
    shares, each alone and then all at once, beside a thread whose launches
    hold the device most of the time."""
    ss = [cancelling((47, 44, 40 + k), 1 + k) for k in range(3)]
    ctxs = [context(s) for s in ss]
    bs = [cancelling((40, 38, 35), 9), cancelling((46, 44, 30), 10)]
    bt = batch(bs)
    for _ in range(2):
        loop = [solve(c, s, -1) for c, s in zip(ctxs, ss)]
    alone = [solve(c, s) for c, s in zip(ctxs, ss)]
    # (the two orders are told apart)
    assert not any(np.array_equal(a, b, equal_nan=True) for a, b in zip(alone, loop))
    alone_b = batch_solve(bt, bs)
    busy = mesh.varcoeff3d((64, 64, 64), seed=11, permute=False)
    cb = context(busy)
    over = threading.Event()

    def long_solve():
        cb.solve(_lib.CF_SOLVER_PCG, np.zeros(busy.n), busy.source,
                 _lib.default_options(tolerance=1e-30, maxIter=400, maxRestarts=0))

    def keep_busy():
        while not over.is_set():
            long_solve()

    for _ in range(3):
        long_solve()
    keep_busy_thread = threading.Thread(target=keep_busy)
    keep_busy_thread.start()
    out = [[] for _ in range(4)]

    def work(k):
        for _ in range(12):
            out[k].append(solve(ctxs[k], ss[k]) if k < 3 else batch_solve(bt, bs))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    over.set()
    keep_busy_thread.join()
    cb.close()
    for k in range(3):
        assert len(out[k]) == 12
        assert all(np.array_equal(x, alone[k], equal_nan=True) for x in out[k]), k
        ctxs[k].close()
    assert len(out[3]) == 12
    for xs in out[3]:
        assert all(np.array_equal(x, a, equal_nan=True) for x, a in zip(xs, alone_b))
    bt.close()


def many(ctxs, ss, solver, opts):
    import torch
    xs = [torch.zeros(s.n, dtype=torch.float64, device="cuda") for s in ss]
    bs = [torch.from_numpy(s.source).cuda() for s in ss]
    torch.cuda.synchronize()
    l0 = [c.kernel_launches() for c in ctxs]
    p = _lib.solve_many_device(ctxs, solver, xs, bs, opts, streams=8)
    return [x.cpu().numpy() for x in xs], [c.kernel_launches() - n for c, n in zip(ctxs, l0)], p


# rows per SM at both ends of the range that leaves cudaPCG to graph loops
# with four systems at once, and three systems
@pytest.mark.parametrize("rows,count,split", [(384, 4, True), (385, 4, False), (1216, 4, False),
                                              (1217, 4, True), (600, 3, True)])
def test_many_pcg_takes_one_form(require_gpu, rows, count, split):
    import torch
    m = torch.cuda.get_device_properties(0).multi_processor_count
    ss = [cancelling((m, rows), 20 + k) for k in range(count)]
    ctxs = [context(s) for s in ss]
    for _ in range(2):
        loop = [solve(c, s, -1) for c, s in zip(ctxs, ss)]
    alone = [solve(c, s) for c, s in zip(ctxs, ss)]
    for _ in range(3):
        xs, _, _ = many(ctxs, ss, _lib.CF_SOLVER_PCG, _lib.default_options(**OPTS))
        for x, a, g in zip(xs, alone, loop):
            assert np.array_equal(x, a if split else g, equal_nan=True)
    for c in ctxs:
        c.close()


# momentum systems of two and three 256-row groups per SM and of more than
# 2,560 rows per SM; the same bits in every form, told apart by their launches
@pytest.mark.parametrize("rows,count,form", [(520, 2, "whole"), (520, 3, "loop"),
                                             (2561, 3, "whole")])
def test_many_bicgstab_forms(require_gpu, rows, count, form):
    import torch
    m = torch.cuda.get_device_properties(0).multi_processor_count
    ss = [mesh.upwind3d((m, rows), seed=40 + k) for k in range(count)]
    ctxs = [context(s) for s in ss]
    kw = dict(tolerance=1e-6, maxIter=40, maxRestarts=1)
    ref, loop, _ = many(ctxs, ss, _lib.CF_SOLVER_PBICGSTAB,
                        _lib.default_options(clusterMaxCells=-1, **kw))
    xs, launches, _ = many(ctxs, ss, _lib.CF_SOLVER_PBICGSTAB, _lib.default_options(**kw))
    for x, r, a, b in zip(xs, ref, launches, loop):
        assert np.array_equal(x, r)
        assert (a < b) if form == "whole" else (a == b), (a, b)
    for c in ctxs:
        c.close()


def test_persistent_launches_take_turns(require_gpu):
    """The opt-in persistent inner solves, of a context and of a batch, at the
    same time as solves on the split over the SMs: none runs into its wait
    limit, all results as alone."""
    ss = [mesh.varcoeff3d((40, 40, 22), seed=50, permute=True),
          mesh.varcoeff3d((44, 42, 40), seed=51, permute=True)]
    ctxs = [context(s) for s in ss]
    bs = [mesh.poisson2d(100, 90, seed=52), mesh.varcoeff3d((24, 24, 24), seed=53)]
    bt = batch(bs)

    def opts(persistent):
        return _lib.default_options(persistentMaxCells=1000000 if persistent else 0, maxIter=200)

    def one(k):
        if k < 2:
            x = np.zeros(ss[k].n)
            ctxs[k].solve(_lib.CF_SOLVER_PCG, x, ss[k].source, opts(k == 0))
            return [x]
        xs = [np.zeros(s.n) for s in bs]
        bt.solve(xs, [s.source for s in bs], opts(True))
        return xs

    for _ in range(3):
        alone = [one(k) for k in range(3)]
    out = [[] for _ in range(3)]

    def work(k):
        for _ in range(8):
            out[k].append(one(k))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(3):
        assert len(out[k]) == 8
        for xs in out[k]:
            assert all(np.array_equal(x, a) for x, a in zip(xs, alone[k])), k
    for c in ctxs:
        c.close()
    bt.close()
