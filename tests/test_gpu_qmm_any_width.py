"""The fp16 streaming kernel: contraction widths that are only multiples of the group size, every group size, row counts and
token counts around its tiles, against the CPU oracle (fp32 weight term)."""
import numpy as np
import pytest
import torch

from oracle import qoracle as qo
from test_gpu_qmm import _run
from util import dev_triple, gate_f32, make_weight, rand_bf16, to_dev_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,gs,M,N,K", [
    (4, 64, 1, 16, 64), (4, 64, 8, 7211, 2880), (8, 64, 5, 65, 576), (4, 64, 3, 1, 14272),         # one group; odd pitches of scales
    (4, 32, 1, 300, 32), (4, 32, 8, 129, 1056), (8, 32, 7, 300, 2016), (8, 128, 4, 63, 1152), (4, 128, 2, 700, 640),
    (4, 64, 9, 515, 2880), (8, 64, 16, 130, 192), (4, 32, 17, 257, 992), (8, 128, 32, 64, 1664),   # two and four token tiles
    (4, 64, 33, 200, 704), (4, 32, 70, 65, 288)])                                                  # more than one pass
def test_any_width(bits, gs, M, N, K):
    rng = np.random.default_rng(bits * 1000 + gs + M + N + K)
    q, s, b = make_weight(rng, (N, K), gs, bits)
    r32, _ = _run(rand_bf16(rng, (M, K)), q, s, b, gs, bits)
    assert r32 < 1e-4


def test_several_matrices_and_wide_ranges():
    """Three matrices in one call (row shares cross their borders); activations over 40 octaves; rows of a larger matrix."""
    import qb200
    rng = np.random.default_rng(3)
    K, M = 1344, 6
    ws = [make_weight(rng, (n, K), 64, 4) for n in (700, 33, 250)]
    x = qo.bf16_round((rng.standard_normal((M, K)) * np.exp2(rng.integers(-20, 20, (M, K)))).astype(np.float32))
    dev = [dev_triple(*w) for w in ws]
    dev[1] = [t[4:28] for t in dev[1]]
    outs = [torch.empty((M, n), dtype=torch.float32, device="cuda") for n in (700, 24, 250)]
    qb200.quantized_matmul_batch(torch.from_numpy(x).cuda(), dev, outs, True, 64, 4)
    for y, w, sl in zip(outs, ws, (slice(None), slice(4, 28), slice(None))):
        gate_f32(y.cpu().numpy(), qo.qmm(x, *[a[sl] for a in w], 64, 4), "several matrices")
    xn = x.copy()
    xn[2, 77] = np.inf
    y = qb200.quantized_matmul(to_dev_bf16(qo.f32_to_bf16(xn)), *dev[0], True, 64, 4)
    assert torch.isnan(y[2]).all() and torch.isfinite(y[[0, 1, 3, 4, 5]]).all()
    assert qb200.lib().qb200_debug_tc_status() == 0


@pytest.mark.parametrize("M,N,K", [(5, 40000, 704), (16, 12000, 8896)])   # several blocks a CTA; a cluster over K, two token tiles
def test_waits_that_run_out(M, N, K):
    """A wait that gives up ends the launch: its status is set, nothing is stored behind it, and the next launch is as ever."""
    import qb200
    L = qb200.lib()
    w = qb200.quantize(torch.randn(N, K, device="cuda", dtype=torch.bfloat16) * 0.02, 64, 4)
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    good = qb200.quantized_matmul(x, *w, True, 64, 4)
    assert L.qb200_debug_tc_status() == 0
    try:
        for polls in (-1, 1, 2):
            y = torch.full_like(good, float("nan"))
            L.qb200_debug_wait_polls(polls)
            qb200.quantized_matmul(x, *w, True, 64, 4, out=y)
            status, done = L.qb200_debug_tc_status(), ~torch.isnan(y)
            assert status in (201, 202, 203, 204, 205) or (polls > 0 and status == 0)
            assert bool((y[done] == good[done]).all())
            assert (status == 0) == bool(done.all())
            assert polls > 0 or not bool(done.any())
            L.qb200_debug_tc_reset()
    finally:
        L.qb200_debug_wait_polls(0)
        L.qb200_debug_tc_reset()
    assert torch.equal(qb200.quantized_matmul(x, *w, True, 64, 4), good)
    assert L.qb200_debug_tc_status() == 0


@pytest.mark.parametrize("bits,gs,M,N,K", [(4, 64, 4, 600, 20096), (8, 128, 4, 300, 19968), (4, 32, 4, 130, 19232)])
def test_a_cluster_over_k_and_where_none_can_be_placed(bits, gs, M, N, K):
    """Activations of that length are split over a cluster; without one the kernels before this one serve them."""
    import qb200
    test_any_width(bits, gs, M, N, K)
    qb200.lib().qb200_debug_refuse_clusters(True)
    try:
        test_any_width(bits, gs, M, N, K)
        rng = np.random.default_rng(K)
        w = [make_weight(rng, (n, K), gs, bits) for n in (N, 33)]
        x = rand_bf16(rng, (M, K))
        y = [torch.empty((M, n), dtype=torch.float32, device="cuda") for n in (N, 33)]
        qb200.quantized_matmul_batch(torch.from_numpy(x).cuda(), [dev_triple(*t) for t in w], y, True, gs, bits)
        for r, t in zip(y, w):
            gate_f32(r.cpu().numpy(), qo.qmm(x, *t, gs, bits), "several matrices")
    finally:
        qb200.lib().qb200_debug_refuse_clusters(False)
