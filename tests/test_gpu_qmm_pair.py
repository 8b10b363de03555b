"""The CTA-pair tensor-core kernel: edges of its token and weight-row tiles, one and two units a tile, several waves, and rows sorted
by expert, against the CPU oracle (weight term rounded to bf16 once)."""
import numpy as np
import pytest
import torch

from oracle import qoracle as qo
from test_gpu_qmm import _run
from util import dev_triple, gate_bf16, make_weight, rand_bf16, to_dev_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,gs,M,N,K", [
    (4, 64, 257, 512, 256), (8, 64, 289, 769, 512), (4, 128, 513, 1023, 768), (4, 64, 129, 6144, 256),   # edges of units and row blocks
    (4, 64, 1000, 600, 1280), (8, 128, 1100, 2304, 256), (4, 64, 2500, 5000, 256)])                      # several waves, one unit and two
def test_dense(bits, gs, M, N, K):
    import qb200
    rng = np.random.default_rng(bits * 100 + gs + M + N + K)
    q, s, b = make_weight(rng, (N, K), gs, bits)
    x = rand_bf16(rng, (M, K))
    if M * N < 1 << 20:
        _run(x, q, s, b, gs, bits)
    else:   # the oracle takes sampled rows
        y = qb200.quantized_matmul(to_dev_bf16(qo.f32_to_bf16(x)), *dev_triple(q, s, b), True, gs, bits).float().cpu().numpy()
        rows = rng.choice(M, 48, replace=False)
        gate_bf16(y[rows], qo.qmm(x[rows], q, s, b, gs, bits, bf16_weights=True), "sampled rows")
    assert qb200.lib().qb200_debug_tc_status() == 0


@pytest.mark.parametrize("bits,gs,N,K,counts", [
    (4, 64, 300, 256, (600, 0, 33, 1, 513, 70)), (8, 64, 256, 512, (0, 257, 900, 31)), (4, 128, 513, 256, (5, 2000)),
    (4, 64, 256, 256, tuple(32 + (i * 7) % 5 for i in range(300)))])                                     # more experts than fit beside six stages
def test_sorted_rows(bits, gs, N, K, counts):
    import qb200
    rng = np.random.default_rng(len(counts) + N + K)
    E = len(counts)
    q, s, b = make_weight(rng, (E, N, K), gs, bits)
    x = rand_bf16(rng, (sum(counts), 1, K))
    idx = np.repeat(np.arange(E), counts).astype(np.int32)
    y = qb200.gather_qmm(to_dev_bf16(qo.f32_to_bf16(x)), *dev_triple(q, s, b), None, torch.from_numpy(idx).cuda(), True, gs, bits, sorted_indices=True)
    x, y = x[:, 0], y.float().cpu().numpy()[:, 0]
    for e in range(0, E, 1 + E // 20):
        if counts[e]:
            gate_bf16(y[idx == e], qo.qmm(x[idx == e], q[e], s[e], b[e], gs, bits, bf16_weights=True), f"expert {e}")
    assert qb200.lib().qb200_debug_tc_status() == 0


@pytest.mark.parametrize("bits", [4, 8])
def test_tile_of_more_than_a_millisecond(bits):
    """One tile over a long contraction: the epilogue waits 2.3 ms.  Checked against the exact sum."""
    import qb200
    M, N, K = 257, 512, 196608
    w = qb200.quantize(torch.randn(N, K, device="cuda", dtype=torch.bfloat16) * 0.02, 64, bits)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    y = qb200.quantized_matmul(x, *w, True, 64, bits)
    assert qb200.lib().qb200_debug_tc_status() == 0
    ref = x[:64].double() @ qb200.dequantize(*w, 64, bits, dtype=torch.bfloat16).double().t()
    assert float((y[:64].double() - ref).norm() / ref.norm()) < 3e-3


@pytest.mark.parametrize("bits", [4, 8])
def test_tile_of_a_tenth_of_a_second(bits):
    """The epilogue waits for more than 2^18 polls.  x is zero but for 96 places over the whole of K, and every product a multiple of 1/2, so
    that the sum is exact: the result differs by its rounding to bf16 alone (2^-8 of the value)."""
    import qb200
    M, N, K = 257, 512, 10485760
    g = torch.Generator(device="cuda").manual_seed(bits)
    codes = torch.randint(-2 ** 31, 2 ** 31 - 1, (N, K * bits // 32), device="cuda", generator=g, dtype=torch.int32)
    scales = 0.5 * torch.randint(1, 3, (N, K // 64), device="cuda", generator=g).to(torch.bfloat16)
    x = torch.zeros(M, K, device="cuda", dtype=torch.bfloat16)
    at = torch.linspace(0, K - 1, 96, device="cuda").long()
    x[:, at] = torch.randint(-8, 9, (M, 96), device="cuda", generator=g).to(torch.bfloat16)
    y = qb200.quantized_matmul(x, codes, scales, torch.zeros_like(scales), True, 64, bits)
    assert qb200.lib().qb200_debug_tc_status() == 0
    q = (codes[:, at * bits // 32] >> (at * bits % 32)) & (2 ** bits - 1)
    ref = x[:, at].double() @ (q * scales[:, at // 64].float()).to(torch.bfloat16).double().t()
    assert bool(((y.double() - ref).abs() <= 2.0 ** -8 * ref.abs()).all())


def test_where_no_cluster_can_be_placed(no_clusters):
    """The one-CTA kernel takes the pairs' place."""
    test_dense(4, 64, 257, 512, 256)
    test_sorted_rows(8, 64, 256, 512, (0, 257, 900, 31))


@pytest.mark.parametrize("bits,counts", [
    (4, (288, 256, 512, 1, 224, 481, 320, 96)), (8, (510, 290, 33, 300)), (4, (270,) * 8)])
def test_accumulators_in_turn(bits, counts):
    """Several tiles a pair, of one and two units, whose accumulators go round the ring of tensor memory in many ways: cut at its end,
    moved to its start, beside those of the tile before.  One expert's weights against the exact sum over all its rows."""
    import qb200
    N, K, E = 11264, 256, len(counts)                       # 44 tiles and more of 256 weight rows an expert
    g = torch.Generator(device="cuda").manual_seed(bits + E)
    w = qb200.quantize(torch.randn(E, N, K, device="cuda", generator=g).to(torch.bfloat16) * 0.05, 64, bits)
    x = torch.randn(sum(counts), 1, K, device="cuda", generator=g).to(torch.bfloat16)
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts)).int().cuda()
    y = qb200.gather_qmm(x, *w, None, idx, True, 64, bits, sorted_indices=True)
    assert qb200.lib().qb200_debug_tc_status() == 0
    for e in range(E):
        m = idx == e
        wd = qb200.dequantize(*(t[e].contiguous() for t in w), 64, bits, dtype=torch.bfloat16).double()
        ref = x[m, 0].double() @ wd.t()
        # bf16 rounding of the result (2^-8), and fp32 sums of 256 products in any order (2^-23 a step)
        tol = 2.0 ** -8 * ref.abs() + 256 * 2.0 ** -23 * (x[m, 0].double().abs() @ wd.abs().t())
        assert bool(((y[m, 0].double() - ref).abs() <= tol).all()), f"expert {e}"


@pytest.mark.parametrize("bits,counts,N", [
    (4, (96, 160, 224, 31, 256, 190, 64, 129), 11264), (8, (200,) * 12, 11104),     # tiles of one unit only; a last tile of 96 weight rows
    (4, (288, 256, 300, 481, 320), 11299), (8, (512, 290, 430), 11040)])            # two units; last tiles of 35 and 32, odd rows of y
def test_accumulators_in_turn_ragged(bits, counts, N):
    sorted_rows_exact(bits, counts, N)


@pytest.mark.parametrize("M,N,K", [(1138, 14147, 256), (2401, 12013, 512), (600, 9001, 768), (700, 8192, 256), (4096, 4096, 512)])
def test_dense_short_contractions(M, N, K):
    """Several tiles a pair that end after few k-blocks, rows of y on and off 4 bytes."""
    sorted_rows_exact(4, (M,), N, K)


def sorted_rows_exact(bits, counts, N, K=256):
    """The same with any number of weight rows and any contraction; a single expert is a dense product."""
    import qb200
    E = len(counts)
    g = torch.Generator(device="cuda").manual_seed(bits + E)
    w = qb200.quantize(torch.randn(E, N, K, device="cuda", generator=g).to(torch.bfloat16) * 0.05, 64, bits)
    x = torch.randn(sum(counts), 1, K, device="cuda", generator=g).to(torch.bfloat16)
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts)).int().cuda()
    if E == 1:
        y = qb200.quantized_matmul(x[:, 0], *(t[0] for t in w), True, 64, bits)[:, None]
    else:
        y = qb200.gather_qmm(x, *w, None, idx, True, 64, bits, sorted_indices=True)
    assert qb200.lib().qb200_debug_tc_status() == 0
    for e in range(E):
        m = idx == e
        wd = qb200.dequantize(*(t[e].contiguous() for t in w), 64, bits, dtype=torch.bfloat16).double()
        ref = x[m, 0].double() @ wd.t()
        # bf16 rounding of the result (2^-8), and fp32 sums of K products in any order (2^-23 a step)
        tol = 2.0 ** -8 * ref.abs() + K * 2.0 ** -23 * (x[m, 0].double().abs() @ wd.abs().t())
        assert bool(((y[m, 0].double() - ref).abs() <= tol).all()), f"expert {e}"
