"""The tiled fp32-weight kernel: dense products over its tile shapes, shares of K and tails, and rows sorted by expert, against the
CPU oracle (fp32 weight term)."""
import numpy as np
import pytest
import torch

from oracle import qoracle as qo
from test_gpu_qmm import _run
from util import dev_triple, make_weight, rand_bf16, to_dev_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,gs,M,N,K", [
    (4, 64, 33, 129, 2880), (4, 64, 9, 300, 4416), (8, 64, 65, 127, 704),    # edges of tiles; long and uneven shares of K
    (4, 32, 40, 260, 1056), (8, 32, 130, 65, 992), (8, 128, 47, 1000, 896),  # half a stage at the end; one scale for two groups
    (4, 64, 6, 515, 3520), (4, 64, 700, 1537, 192), (8, 64, 300, 2100, 320)])  # few tokens; several waves
def test_dense(bits, gs, M, N, K):
    rng = np.random.default_rng(bits * 100 + gs + M + N + K)
    q, s, b = make_weight(rng, (N, K), gs, bits)
    r32, _ = _run(rand_bf16(rng, (M, K)), q, s, b, gs, bits)
    assert r32 < 1e-4


@pytest.mark.parametrize("bits,gs,E,N,K,counts", [
    (4, 64, 5, 130, 192, (3, 0, 17, 1, 40)), (8, 64, 3, 257, 704, (100, 33, 64)), (4, 32, 4, 65, 352, (0, 9, 0, 70)),
    (8, 128, 2, 128, 640, (1, 200)),
    (4, 64, 3, 60, 64, (2500, 1, 1600))])                                    # too many rows for a CTA per piece
def test_sorted_rows(bits, gs, E, N, K, counts):
    import qb200
    rng = np.random.default_rng(E + N + K)
    q, s, b = make_weight(rng, (E, N, K), gs, bits)
    x = rand_bf16(rng, (sum(counts), 1, K))
    idx = np.repeat(np.arange(E), counts).astype(np.int32)
    y = qb200.gather_qmm(to_dev_bf16(qo.f32_to_bf16(x)), *dev_triple(q, s, b), None, torch.from_numpy(idx).cuda(), True, gs, bits, sorted_indices=True)
    xf, y = x[:, 0], y.float().cpu().numpy()[:, 0]
    for e in range(E):
        r = qo.qmm(xf[idx == e], q[e], s[e], b[e], gs, bits)
        rms = np.sqrt(np.mean(r * r, axis=-1, keepdims=True)) + 1e-30
        assert (np.abs(y[idx == e] - r) <= np.abs(r) * 2.0 ** -8 + 1e-4 * rms).all()


@pytest.mark.parametrize("bits,gs,M,N,K", [(4, 64, 9, 300, 4416), (8, 64, 65, 127, 704), (4, 32, 40, 260, 1056)])
def test_where_no_cluster_can_be_placed(no_clusters, bits, gs, M, N, K):
    """A CTA takes the whole of K."""
    test_dense(bits, gs, M, N, K)
