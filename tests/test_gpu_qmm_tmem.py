"""The kernel that streams weights through tensor memory (9 - 64 tokens): edges of its token blocks, row tiles and shares of K, scales on
either side of what its conversion takes at once, several matrices in a call, a device that places no clusters -- against the CPU
oracle (weight term rounded to bf16 once)."""
import numpy as np
import pytest
import torch

from oracle import qoracle as qo
from test_gpu_qmm import _run
from util import dev_triple, gate_bf16, make_weight, rand_bf16, to_dev_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,gs,M,N,K", [
    (4, 64, 9, 1, 256), (4, 64, 16, 127, 512), (4, 128, 17, 128, 768), (4, 64, 32, 129, 1280),      # one row; edges of tiles; scales' rows of 24, 40 bytes
    (4, 64, 33, 300, 2048), (4, 64, 48, 640, 256), (4, 128, 64, 513, 1024), (4, 64, 64, 100, 4352),
    (8, 64, 9, 130, 256), (8, 128, 16, 257, 1792), (8, 64, 27, 64, 3072), (8, 64, 49, 200, 512), (8, 128, 64, 129, 768),
    (4, 64, 13, 20000, 256), (8, 64, 32, 9000, 512), (8, 64, 32, 30000, 512),                       # (on 148 SMs) two tiles a CTA, one, two
    (4, 64, 20, 256, 16384), (8, 64, 64, 140, 8192)])                                               # x in a ring
def test_edges(bits, gs, M, N, K):
    import qb200
    rng = np.random.default_rng(bits * 100 + gs + M + N + K)
    q, s, b = make_weight(rng, (N, K), gs, bits)
    _run(rand_bf16(rng, (M, K)), q, s, b, gs, bits)
    assert qb200.lib().qb200_debug_tc_status() == 0


@pytest.mark.parametrize("bits,gs,M,N,K", [(4, 64, 12, 500, 16640), (8, 64, 32, 300, 20480), (4, 128, 20, 400, 28672), (8, 128, 9, 100, 16640), (4, 64, 33, 200, 16640)])
def test_long_contractions(bits, gs, M, N, K):
    """Above 16384 the weight term is fp32 up to 32 tokens, but at 8 bits of groups of 128; alone and two matrices in a call."""
    import qb200
    rng = np.random.default_rng(M + N + K)
    q, s, b = make_weight(rng, (N, K), gs, bits)
    x = rand_bf16(rng, (M, K))
    _run(x, q, s, b, gs, bits)
    dw, dx = dev_triple(q, s, b), to_dev_bf16(qo.f32_to_bf16(x))
    outs = [torch.empty((M, N), dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    qb200.quantized_matmul_batch(dx, [dw, dw], outs, True, gs, bits)
    for y in outs:
        gate_bf16(y.float().cpu().numpy(), qo.qmm(x, q, s, b, gs, bits, bf16_weights=M > 32 or gs * bits == 1024), "two matrices")


@pytest.mark.parametrize("bits", [4, 8])
def test_scales_of_all_sizes(bits):
    """Groups from 2^-30 to 2^30: those that the conversion of codes as subnormals takes, those beyond, and both in a unit."""
    import qb200
    rng = np.random.default_rng(bits)
    M, N, K = 24, 256, 1024
    w = rand_bf16(rng, (N, K)) * np.exp2(rng.integers(-30, 31, (N, K // 64))).astype(np.float32).repeat(64, 1)
    w[:128] = rand_bf16(rng, (128, K), 0.02)
    w[5, 64:128] = 1000.0 * rand_bf16(rng, (64,))
    q, s, b = qo.quantize(w, 64, bits)
    x = rand_bf16(rng, (M, K))
    y = qb200.quantized_matmul(to_dev_bf16(qo.f32_to_bf16(x)), *dev_triple(q, s, b), True, 64, bits).float().cpu().numpy()
    ref = qo.qmm(x, q, s, b, 64, bits, bf16_weights=True)
    for n in range(N):   # (a row's own size)
        gate_bf16(y[:, n], ref[:, n], f"row {n}")


def test_several_matrices():
    import qb200
    rng = np.random.default_rng(5)
    K, M, rows = 1024, 19, (700, 33, 128, 250)
    ws = [make_weight(rng, (n, K), 64, 4) for n in rows]
    x = rand_bf16(rng, (M, K))
    dev, dx = [dev_triple(*w) for w in ws], to_dev_bf16(qo.f32_to_bf16(x))
    outs = [torch.empty((M, n), dtype=torch.bfloat16, device="cuda") for n in rows]
    qb200.quantized_matmul_batch(dx, dev, outs, True, 64, 4)
    for y, w, d in zip(outs, ws, dev):
        gate_bf16(y.float().cpu().numpy(), qo.qmm(x, *w, 64, 4, bf16_weights=True), "several matrices")
    qb200.lib().qb200_debug_refuse_clusters(True)
    try:
        alone = qb200.quantized_matmul(dx, *dev[0], True, 64, 4)
    finally:
        qb200.lib().qb200_debug_refuse_clusters(False)
    gate_bf16(alone.float().cpu().numpy(), qo.qmm(x, *ws[0], 64, 4, bf16_weights=True), "no clusters")
    assert qb200.lib().qb200_debug_tc_status() == 0


def _weight(n, k, gs, bits, g):
    import qb200
    return qb200.quantize((torch.randn((n, k), device="cuda", generator=g) * 0.02).to(torch.bfloat16), gs, bits)


def _gate_exact(y, x, w, gs, bits, what):
    """Every output against the 64-bit sum: the rounding of the result to bf16 (2^-8 of it at most), and fp32 sums of K products in any
    order (2^-23 a step)."""
    import qb200
    wd, xd = qb200.dequantize(*w, gs, bits, dtype=torch.bfloat16).double(), x.double()
    ref = xd @ wd.t()
    tol = 2.0 ** -8 * ref.abs() + x.shape[1] * 2.0 ** -23 * (xd.abs() @ wd.abs().t())
    bad = ~((y.double() - ref).abs() <= tol)
    assert not bool(bad.any()), f"{what}: {int(bad.sum())} of {bad.numel()}"


# (on 148 SMs: tiles of 128 rows, the CTAs that share a row tile, units of K of one)
@pytest.mark.parametrize("bits,gs,M,N,K", [
    (4, 64, 9, 19500, 256), (4, 64, 32, 40000, 256), (8, 64, 17, 40000, 256), (4, 128, 64, 40000, 256),    # 1 CTA, 1 unit: the second group's first one is in the second tile
    (4, 64, 16, 40000, 768), (8, 128, 32, 19500, 1280), (4, 64, 25, 10000, 8192),                          # odd shares: units change groups from tile to tile
    (4, 64, 25, 11264, 2560)])                                                                             # a tile a CTA
def test_activations_of_the_kernel_before(bits, gs, M, N, K):
    """Two linears in a graph, the first one's output the second one's activations: the second is let in early and converts its weights
    meanwhile, and has to wait for every unit of x."""
    import qb200
    g = torch.Generator(device="cuda").manual_seed(N + K + M)
    w1, w2 = _weight(K, 14336, 64, 4, g), _weight(N, K, gs, bits, g)
    x = torch.randn((M, 14336), device="cuda", generator=g).to(torch.bfloat16)
    h, y = (torch.zeros((M, n), dtype=torch.bfloat16, device="cuda") for n in (K, N))

    def chain():
        qb200.quantized_matmul(x, *w1, True, 64, 4, out=h)
        qb200.quantized_matmul(h, *w2, True, gs, bits, out=y)

    chain()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain()
    for i in range(5):
        x.copy_(torch.randn(x.shape, device="cuda", generator=g))
        torch.cuda.synchronize()
        graph.replay()
        _gate_exact(h, x, w1, 64, 4, f"first, replay {i}")
        _gate_exact(y, h, w2, gs, bits, f"second, replay {i}")
    assert qb200.lib().qb200_debug_tc_status() == 0


@pytest.mark.parametrize("M", [16, 32, 64])
@pytest.mark.parametrize("bits,gs,N,K", [
    (4, 64, 28672, 4096), (8, 64, 13000, 4096), (4, 128, 11648, 2560), (4, 64, 12000, 2304),   # CTAs by themselves
    (4, 64, 19200, 8192),                                                                      # clusters of four, five tiles each
    (4, 128, 10000, 8192), (8, 64, 10000, 8192)])                                              # of three, two tiles: shares of 10, 11, 11 units
def test_several_tiles_a_cluster(bits, gs, N, K, M):
    import qb200
    g = torch.Generator(device="cuda").manual_seed(N + K + M)
    w = _weight(N, K, gs, bits, g)
    x = torch.randn((M, K), device="cuda", generator=g).to(torch.bfloat16)
    y = qb200.quantized_matmul(x, *w, True, gs, bits)
    _gate_exact(y, x, w, gs, bits, f"{M} x {N} x {K}")
    assert torch.equal(qb200.quantized_matmul(x, *w, True, gs, bits), y)   # the order of the sum does not depend on timing
    assert qb200.lib().qb200_debug_tc_status() == 0


@pytest.mark.parametrize("bits,gs", [(4, 64), (8, 64), (4, 128)])
@pytest.mark.parametrize("M,N,K", [(9, 130, 256), (16, 640, 1280), (20, 1000, 2048), (32, 300, 4352)])
def test_activations_off_16_bytes(bits, gs, M, N, K):
    """Rows of x that no tensor map takes: the wide streaming kernel, alone and two matrices in a call."""
    import qb200
    rng = np.random.default_rng(M + N + K)
    ws = [make_weight(rng, (n, K), gs, bits) for n in (N, 77)]
    x = rand_bf16(rng, (M, K + 5))
    dx, dev = to_dev_bf16(qo.f32_to_bf16(x))[:, 3:K + 3], [dev_triple(*w) for w in ws]
    refs = [qo.qmm(np.ascontiguousarray(x[:, 3:K + 3]), *w, gs, bits, bf16_weights=True) for w in ws]
    gate_bf16(qb200.quantized_matmul(dx, *dev[0], True, gs, bits).float().cpu().numpy(), refs[0], "alone")
    outs = [torch.empty((M, n), dtype=torch.bfloat16, device="cuda") for n in (N, 77)]
    qb200.quantized_matmul_batch(dx, dev, outs, True, gs, bits)
    for y, ref in zip(outs, refs):
        gate_bf16(y.float().cpu().numpy(), ref, "two matrices")
    assert qb200.lib().qb200_debug_tc_status() == 0


@pytest.mark.parametrize("M", [9, 32])
def test_rows_that_no_tensor_map_takes(M):
    """Broadcast and overlapping rows of x, of the weights and of their scales, and a single row of a pitch beyond a map's."""
    import qb200
    rng = np.random.default_rng(M)
    N, K = 200, 512
    w, x = make_weight(rng, (N, K), 64, 4), rand_bf16(rng, (M, K))
    dev, dx, flat = dev_triple(*w), to_dev_bf16(qo.f32_to_bf16(x)), rand_bf16(rng, (K + 8 * M,))
    slid = np.stack([flat[8 * i:8 * i + K] for i in range(M)])
    cases = {
        "x of one row": (dx[:1].expand(M, K), dev, x[:1].repeat(M, 0), w),
        "x as windows": (to_dev_bf16(qo.f32_to_bf16(flat)).as_strided((M, K), (8, 1)), dev, slid, w),
        "weights of one row": (dx, [t[:1].expand(N, t.shape[1]) for t in dev], x, [t[:1].repeat(N, 0) for t in w]),
        "scales of one row": (dx, [dev[0]] + [t[:1].expand(N, t.shape[1]) for t in dev[1:]], x, [w[0]] + [t[:1].repeat(N, 0) for t in w[1:]]),
        "one row, no pitch": (dx, [t.as_strided((1, t.shape[1]), (0, 1)) for t in dev], x, [t[:1] for t in w]),
        "one row, any pitch": (dx, [t.as_strided((1, t.shape[1]), (1 << 40, 1)) for t in dev], x, [t[:1] for t in w]),
    }
    for what, (xd, wd, xh, wh) in cases.items():
        ref = qo.qmm(np.ascontiguousarray(xh), *[np.ascontiguousarray(t) for t in wh], 64, 4, bf16_weights=True)
        gate_bf16(qb200.quantized_matmul(xd, *wd, True, 64, 4).float().cpu().numpy(), ref, what)
        outs = [torch.empty((M, ref.shape[1]), dtype=torch.bfloat16, device="cuda") for _ in range(2)]
        qb200.quantized_matmul_batch(xd, [wd, wd], outs, True, 64, 4)
        for y in outs:
            gate_bf16(y.float().cpu().numpy(), ref, what + ", twice")
    assert qb200.lib().qb200_debug_tc_status() == 0


@pytest.mark.parametrize("bits,M,N,K", [
    (4, 16, 10000, 8192), (4, 64, 19200, 8192),      # clusters with several tiles
    (4, 16, 28672, 4096), (4, 64, 11648, 2560), (4, 13, 40000, 768), (8, 64, 300, 8192)])   # CTAs by themselves; x in a ring
def test_waits_that_run_out(bits, M, N, K):
    """A wait that gives up ends the launch: its status is set, nothing is stored behind it, and the next launch is as ever."""
    import qb200
    L = qb200.lib()
    g = torch.Generator(device="cuda").manual_seed(N + K + M)
    w = _weight(N, K, 64, bits, g)
    x = torch.randn((M, K), device="cuda", generator=g).to(torch.bfloat16)
    good = qb200.quantized_matmul(x, *w, True, 64, bits)
    assert L.qb200_debug_tc_status() == 0
    try:
        for polls in (-1, 1, 2, 5):
            y = torch.full_like(good, float("nan"))
            L.qb200_debug_wait_polls(polls)
            qb200.quantized_matmul(x, *w, True, 64, bits, out=y)
            status, done = L.qb200_debug_tc_status(), ~torch.isnan(y)
            assert status in (401, 403, 404, 405, 407) or (polls > 0 and status == 0)
            assert bool((y[done] == good[done]).all())
            assert (status == 0) == bool(done.all())
            assert polls > 0 or not bool(done.any())
            L.qb200_debug_tc_reset()
    finally:
        L.qb200_debug_wait_polls(0)
        L.qb200_debug_tc_reset()
    assert torch.equal(qb200.quantized_matmul(x, *w, True, 64, bits), good)
    assert L.qb200_debug_tc_status() == 0
