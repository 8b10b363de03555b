"""Arguments that the Python functions refuse, by an exception and without a GPU."""
import pytest
import torch

import qb200

BF16 = torch.bfloat16


def triple(*lead):
    """(codes, scales, biases) of rows of 128 values at 4 bits."""
    return torch.zeros(*lead, 16, dtype=torch.int32), torch.zeros(*lead, 2, dtype=BF16), torch.zeros(*lead, 2, dtype=BF16)


def attention(bits, **kw):
    return qb200.kv_decode_attention(torch.zeros(1, 4, 1, 128, dtype=BF16), triple(1, 2, 8), triple(1, 2, 8), bits, 64, 0.1, **kw)


def attention_ptrs(bits, **kw):
    return qb200.kv_decode_attention_ptrs(torch.zeros(2, 4, 1, 128, dtype=BF16), [triple(1, 2, 8)] * 2, [triple(1, 2, 8)] * 2, bits, 64, 0.1, **kw)


@pytest.mark.parametrize("call", [
    lambda: qb200.dequantize(*triple(4), 64, 0),
    lambda: qb200.quantize(torch.zeros(4, 128, dtype=BF16), 0, 4),
    lambda: attention(0),
    lambda: attention(0, out=torch.zeros(1, 4, 1, 128, dtype=BF16), workspace=torch.zeros(1024, dtype=torch.uint8)),
    lambda: attention_ptrs(0),
    lambda: attention_ptrs(0, out=torch.zeros(2, 4, 1, 128, dtype=BF16)),
], ids=["dequantize", "quantize_gs", "attention", "attention_out", "attention_ptrs", "attention_ptrs_out"])
def test_a_size_divided_by_zero(call):
    with pytest.raises(ZeroDivisionError):
        call()


@pytest.mark.parametrize("call", [
    lambda: qb200.dequantize(*triple(4), 64, -4),
    lambda: qb200.quantize(torch.zeros(4, 128, dtype=BF16), -64, 4),
    lambda: attention(-4),
    lambda: attention_ptrs(-4),
    lambda: qb200.dequantize(*triple(4), 64, 2 ** 40),   # (0 values a row; no 32-bit number)
], ids=["dequantize", "quantize_gs", "attention", "attention_ptrs", "dequantize_large"])
def test_sizes_that_no_tensor_has(call):
    with pytest.raises((RuntimeError, OverflowError)):
        call()


@pytest.mark.parametrize("call", [
    lambda: qb200.dequantize(*triple(4), 64, 4.0),
    lambda: qb200.quantize(torch.zeros(4, 128, dtype=BF16), 64, 4.0),
    lambda: attention(4.0),
], ids=["dequantize", "quantize", "attention"])
def test_sizes_are_whole_numbers(call):
    with pytest.raises(TypeError):
        call()


def test_a_cache_is_three_tensors():
    for bad in (triple(1, 2, 8)[:2], triple(1, 2, 8) + (None,)):
        with pytest.raises(ValueError):
            qb200.kv_decode_attention(torch.zeros(1, 4, 1, 128, dtype=BF16), bad, triple(1, 2, 8), 4, 64, 0.1)


@pytest.mark.parametrize("sequences", [0, 2])
@pytest.mark.parametrize("k, v", [(0, 0), (1, 2), (2, 1), (3, 2), (2, 3)])
def test_lists_are_as_long_as_the_batch(sequences, k, v):
    """(a batch of none read the first entry of an empty list)"""
    q = torch.zeros(sequences, 4, 1, 128, dtype=BF16)
    with pytest.raises(IndexError):
        qb200.kv_decode_attention_ptrs(q, [triple(1, 2, 8)] * k, [triple(1, 2, 8)] * v, 4, 64, 0.1)


@pytest.mark.parametrize("dims", [(), (8,)])
def test_cache_views_have_heads_and_tokens(dims):
    q = torch.zeros(1, 4, 1, 128, dtype=BF16)
    with pytest.raises(IndexError):
        qb200.kv_decode_attention_ptrs(q, [triple(*dims)], [triple(1, 2, 8)], 4, 64, 0.1)


@pytest.mark.parametrize("v, offsets", [(3, 2), (2, 3), (1, 2), (2, 1)])
def test_appended_sequences(v, offsets):
    dense = torch.zeros(2, 2, 1, 128, dtype=BF16)
    with pytest.raises(IndexError):
        qb200.kv_append_seqs([triple(1, 2, 8)] * 2, [triple(1, 2, 8)] * v, dense, dense, [0] * offsets, 4, 64)


def test_matrices_and_results():
    x, y = torch.zeros(1, 128, dtype=BF16), torch.zeros(1, 4, dtype=BF16)
    for n in (1, 3):
        with pytest.raises(IndexError):
            qb200.quantized_matmul_batch(x, [triple(4)] * 2, [y] * n, True, 64, 4)


def test_slots_per_token_are_a_whole_number():
    with pytest.raises(TypeError):
        qb200.moe_route(torch.zeros(2, 8), 2.0)
