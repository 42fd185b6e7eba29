"""The allocation-free SpMV + dot: calls that overlap against its contract
spoil their own dot products and no later one, and rows with every number of
faces around the three per side that are loaded together."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Call:
    """One call on device arrays of a mesh; its dot product lands in .dot."""

    def __init__(self, addr, diag, upper, lower, x, w):
        import torch
        arrays = (diag, upper, lower, *addr.arrays(), x, w)
        self.dev = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in arrays]
        self.n = addr.n
        self.y = torch.empty(addr.n, dtype=torch.float32, device="cuda")
        self.dot = torch.zeros(1, dtype=torch.float64, device="cuda")

    def __call__(self, stream=None):
        import torch

        from metal4foam_b200 import _lib
        s = stream or torch.cuda.current_stream()
        _lib.check(_lib.load().cf_ldu_spmv_dot_noalloc(
            self.n, *(_lib.ptr(t) for t in self.dev), _lib.ptr(self.y), _lib.ptr(self.dot),
            _lib.vp(s.cuda_stream)))


def test_overlapping_calls_spoil_no_later_one(require_gpu):
    """A replay of a captured call and, at the same time and against the
    contract, a call that is 32 or 64 calls (the counters of a round) after the
    capture or the last such call; then one call at a time."""
    import torch

    from metal4foam_b200 import mesh
    s = mesh.poisson2d(1500, 1400, seed=1)
    rng = np.random.default_rng(2)
    x, w = (rng.standard_normal(s.n).astype(np.float32) for _ in range(2))
    d, u = s.diag.astype(np.float32), s.upper.astype(np.float32)
    call = Call(s.addr, d, u, u, x, w)
    other = Call(s.addr, d, u, u, x, w)
    call()                                     # (the first call is not captured)
    torch.cuda.synchronize()
    ref = call.dot.item()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=a):
        call(a)
    for _ in range(12):
        for _ in range(31):
            other(b)
        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            graph.replay()
        other(b)
        torch.cuda.synchronize()
    for k in range(200):
        for c, run in ((call, graph.replay), (other, other)):
            c.dot.fill_(float("nan"))
            c.dev[-1].mul_(-2.0 if k % 2 == 0 else -0.5)   # (w: no partial sum is the last one's)
            run()
            torch.cuda.synchronize()
            assert c.dot.item() == (-2.0 * ref if k % 2 == 0 else ref), k


def test_rows_with_every_number_of_faces(require_gpu):
    """0 to 7 faces on the owner side and, on other cells, on the neighbour
    side, against a row-by-row FP32 sum in the call's order."""
    from metal4foam_b200 import mesh
    rng = np.random.default_rng(5)
    pairs, cells, n = set(), 0, 4000
    for width in range(8):                     # cell with `width` cells after it, and before it
        for _ in range(5):
            pairs |= {(cells, cells + k) for k in range(1, width + 1)}
            cells += width + 1
            pairs |= {(cells + k, cells + width) for k in range(width)}
            cells += width + 1
    key = np.array(sorted(pairs), np.int64)
    addr = mesh.ldu_addressing(n, key[:, 0].astype(np.int32), key[:, 1].astype(np.int32))
    assert set(range(8)) <= set(np.diff(addr.ownerStartAddr))
    assert set(range(8)) <= set(np.diff(addr.losortStartAddr))
    diag, x, w = (rng.standard_normal(n).astype(np.float32) for _ in range(3))
    upper, lower = (rng.standard_normal(addr.nf).astype(np.float32) for _ in range(2))
    y = diag * x
    for i in range(n):
        for f in range(addr.ownerStartAddr[i], addr.ownerStartAddr[i + 1]):
            y[i] = np.float32(y[i] + upper[f] * x[addr.upperAddr[f]])
        for k in range(addr.losortStartAddr[i], addr.losortStartAddr[i + 1]):
            f = addr.losortAddr[k]
            y[i] = np.float32(y[i] + lower[f] * x[addr.lowerAddr[f]])
    call = Call(addr, diag, upper, lower, x, w)
    call()
    assert np.array_equal(call.y.cpu().numpy(), y)
    ref = float(w.astype(np.float64) @ y.astype(np.float64))
    # (n terms of magnitude |w y| summed in FP64)
    assert abs(call.dot.item() - ref) <= 1e-13 * np.abs(w * y).sum()
