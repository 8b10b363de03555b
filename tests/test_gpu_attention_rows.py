"""The fp16 tensor-core attention kernel (head dim 64 / 128, GQA up to 8, up to 8 query positions) at the edges of its tiles
and of its dispatch, against the CPU oracle."""
import numpy as np
import pytest
import torch

from oracle import qoracle as qo
from test_gpu_kv_attention import _cache, _run
from util import dev_triple, gate_bf16, gate_f32, rand_bf16, to_dev_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,Hkv,D,bits,T,start", [
    (7, 1, 128, 8, 1, 0), (8, 1, 128, 4, 63, 0), (16, 2, 64, 4, 64, 8), (10, 2, 64, 8, 65, 3),   # one block; odd view starts
    (5, 1, 128, 4, 257, 1), (64, 8, 64, 4, 1000, 0), (12, 2, 128, 8, 4099, 0),
    (8, 1, 128, 4, 20000, 5)])                                                                   # beyond 8 splits: the merge launch
def test_heads_dims_and_lengths(Hq, Hkv, D, bits, T, start):
    _run(np.random.default_rng(Hq + T + bits), 1, Hq, Hkv, T, D, bits, cap=T + start + 7, start=start)


def test_ragged_batch_and_mask():
    rng = np.random.default_rng(5)
    _run(rng, 4, 12, 2, 500, 128, 4, cap=600, lens=[500, 0, 65, 1])
    mask = np.zeros((3, 333), np.float32)
    mask[:, ::7] = -np.inf
    mask[1, :50] = -2.5
    _run(rng, 3, 16, 2, 333, 64, 8, cap=512, mask=mask)


@pytest.mark.parametrize("Hq,Hkv,D,bits,T,Tq", [(28, 4, 128, 8, 700, 4), (8, 8, 64, 4, 8, 8), (16, 2, 128, 4, 1025, 5), (3, 1, 128, 4, 66, 3)])
def test_query_positions(Hq, Hkv, D, bits, T, Tq):
    """Query position tq sees the first T - T_q + 1 + tq cache positions; the positions fill several query tiles."""
    import qb200
    rng = np.random.default_rng(Hq * 10 + T)
    B = 2
    kt, vt = _cache(rng, B, Hkv, T + 9, D, bits)
    q = rand_bf16(rng, (B, Hq, Tq, D))
    kv, vv = [a[:, :, :T] for a in kt], [a[:, :, :T] for a in vt]
    ref = np.stack([qo.kv_decode_attention(q[:, :, i], *kv, *vv, 64, bits, D ** -0.5, kv_lens=[T - Tq + 1 + i] * B) for i in range(Tq)], axis=2)
    dk, dv = ([t[:, :, :T] for t in dev_triple(*c)] for c in (kt, vt))
    o32 = qb200.kv_decode_attention(torch.from_numpy(q).cuda(), dk, dv, bits, 64, D ** -0.5, "causal")
    gate_f32(o32.cpu().numpy(), ref, "fp32 q")
    o16 = qb200.kv_decode_attention(to_dev_bf16(qo.f32_to_bf16(q)).view(B, Hq, Tq, D), dk, dv, bits, 64, D ** -0.5, "causal")
    gate_bf16(o16.float().cpu().numpy(), ref, "bf16 q", slack=4e-3)
