"""Weights that the kernel directly before a linear has written: the linears are programmatic dependents, which start before that kernel's
writes are visible, so they read none of them early unless the host can see what comes before."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def settled():
    import qb200
    return qb200.lib().qb200_debug_weights_settled(C.c_void_p(torch.cuda.current_stream().cuda_stream))


def test_what_the_host_can_see():
    import qb200
    w = qb200.quantize(torch.randn(512, 1024, device="cuda", dtype=BF16), 64, 4)
    r = qb200.quantize(torch.randn(3000, 1088, device="cuda", dtype=BF16), 64, 4)
    cache = [t.view(1, 4, 128, -1) for t in w]   # [1, 4 heads, 128 tokens, 1024]
    norm = torch.ones(1024, device="cuda", dtype=BF16)
    x1, x20, xr = (torch.randn(m, k, device="cuda", dtype=BF16) for m, k in ((1, 1024), (20, 1024), (5, 1088)))
    q = torch.randn(1, 4, 1, 1024, device="cuda", dtype=BF16)
    writes = [lambda: qb200.quantize(x20, 64, 4), lambda: x20.add_(1), lambda: x20.clone(), lambda: w[0].bitwise_not_(),
              lambda: qb200.kv_append(*cache, q, 3, 4, 64)]
    reads = [lambda: qb200.quantized_matmul(x1, *w, True, 64, 4), lambda: qb200.quantized_matmul(x20, *w, True, 64, 4),
             lambda: qb200.quantized_matmul(xr, *r, True, 64, 4), lambda: qb200.rms_norm(x1, norm, 1e-5), lambda: qb200.swiglu(x1, x1)]
    for f in writes + reads:   # first uses, outside a capture
        f()
        assert not settled()
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.graph(torch.cuda.CUDAGraph()):
        assert settled()       # nothing before
        for f in reads:
            f()
            assert settled()
        for f in writes:
            f()
            assert not settled()
            reads[0]()
            assert settled()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            x20.add_(1)
        reads[0]()
        assert settled()
        torch.cuda.current_stream().wait_stream(side)
        assert not settled()   # behind two, one of them unknown


@pytest.mark.parametrize("M,N,K", [(1, 4096, 4096), (8, 4096, 4096), (5, 3000, 2880), (20, 4096, 4096)])
@pytest.mark.parametrize("graph", [False, True])
def test_written_by_the_kernel_before(graph, M, N, K):
    """The codes change under a kernel of torch right before every product, the scales under another."""
    import qb200
    w = qb200.quantize(torch.randn(N, K, device="cuda", dtype=BF16) * 0.02, 64, 4)
    x = torch.randn(M, K, device="cuda", dtype=BF16)
    flip = torch.randint(-2 ** 31, 2 ** 31 - 1, w[0].shape, device="cuda", dtype=torch.int32)
    want = []
    for _ in range(4):
        torch.bitwise_xor(w[0], flip, out=w[0])
        torch.cuda.synchronize()
        want.append(qb200.quantized_matmul(x, *w, True, 64, 4))
        w[1].neg_(), w[2].neg_()
        torch.cuda.synchronize()
        want.append(qb200.quantized_matmul(x, *w, True, 64, 4))
    got = [torch.empty_like(want[0]) for _ in want]

    def chain():
        for i in range(0, len(got), 2):
            torch.bitwise_xor(w[0], flip, out=w[0])
            qb200.quantized_matmul(x, *w, True, 64, 4, out=got[i])
            torch.neg(w[2], out=w[2])
            torch.neg(w[1], out=w[1])
            qb200.quantized_matmul(x, *w, True, 64, 4, out=got[i + 1])

    if graph:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            chain()
    for _ in range(10):
        for y in got:
            y.zero_()
        g.replay() if graph else chain()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
