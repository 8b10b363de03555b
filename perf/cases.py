"""What a host of qb200 has the library do, as cases that can be timed: single quantized linears, the projections of a
decode step, prompt processing, attention over the packed KV cache, a whole decode tick, routed-expert blocks and the
quantize / dequantize work of the cache itself.

A case is a dict of plain values; ``kind`` picks the path.  Sizes are those of this repository's benchmark
configurations (a Llama-3-8B-shaped layer, 128 experts top-8 of 2048 x 768, a 16-sequence cache of 32k tokens) and of
its tests, and around them generic ones: widths that are only multiples of the group size, odd row counts, ragged
lengths.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("mlx-serve_b200"))
import qb200  # noqa: E402

BF16 = torch.bfloat16


def listed():
    return [
        # The smallest thing a host asks for: one linear, one token, one call.  Latency of a call and of a launch.
        {"name": "linear_1_token", "kind": "linear", "M": 1, "N": 4096, "K": 4096, "bits": 4, "gs": 64},
        # A few tokens through a width that is a multiple of the group size only, with an odd number of rows (a
        # vocabulary or a model whose hidden size is no power of two).
        {"name": "linear_5_ragged", "kind": "linear", "M": 5, "N": 7211, "K": 2880, "bits": 4, "gs": 64},
        # Prompt processing: a 2048-token chunk through the widest projection of the layer.
        {"name": "linear_2048_prefill", "kind": "linear", "M": 2048, "N": 14336, "K": 4096, "bits": 4, "gs": 64},
        # The seven projections of a layer, four layers deep, replayed as a CUDA graph (the part of a decode step whose
        # arguments do not change from token to token): one user, eight users, a ragged batch between the kernels'
        # usual widths.
        {"name": "layers_1_token", "kind": "layers", "M": 1, "layers": 4, "hidden": 4096, "kv": 1024, "ffn": 14336, "bits": 4, "gs": 64},
        {"name": "layers_8_tokens", "kind": "layers", "M": 8, "layers": 4, "hidden": 4096, "kv": 1024, "ffn": 14336, "bits": 4, "gs": 64},
        {"name": "layers_27_tokens", "kind": "layers", "M": 27, "layers": 4, "hidden": 4096, "kv": 1024, "ffn": 14336, "bits": 4, "gs": 64},
        # Decode attention of 16 sequences of up to 32k tokens: the largest read of the KV cache.
        {"name": "attention_32k", "kind": "attention", "B": 16, "Hq": 32, "Hkv": 8, "D": 128, "T": 32768, "Tq": 1, "bits": 4, "gs": 64},
        # Verifying four drafted tokens of two sequences, seven query heads to a cache head, 8-bit cache, odd length.
        {"name": "attention_verify", "kind": "attention", "B": 2, "Hq": 28, "Hkv": 4, "D": 128, "T": 4099, "Tq": 4, "bits": 8, "gs": 64},
        # One layer of a continuous-batching tick, call by call (positions change every token, so it is not a graph):
        # 13 sequences, each with a cache of its own and a length of its own.
        {"name": "tick_13_seqs", "kind": "tick", "N": 13, "T": 4000, "hidden": 4096, "Hq": 32, "Hkv": 8, "ffn": 14336, "bits": 4, "gs": 64},
        # The routed-expert block: router, sort, gate / up, SwiGLU, down, weighted sum.  A decode batch and a prompt.
        {"name": "moe_64_tokens", "kind": "moe", "T": 64, "E": 128, "topk": 8, "H": 2048, "I": 768, "bits": 4, "gs": 64},
        {"name": "moe_4096_tokens", "kind": "moe", "T": 4096, "E": 128, "topk": 8, "H": 2048, "I": 768, "bits": 4, "gs": 64},
        # A prompt's keys and values quantized into the cache and read back dense (what a prefill over a cached prefix
        # does before its matrix products).
        {"name": "cache_4096_tokens", "kind": "cache", "B": 2, "Hkv": 8, "D": 128, "S": 4096, "offset": 129, "bits": 8, "gs": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "layers", "layers", "attention", "attention", "tick", "moe", "moe", "cache"])
    bits = rng.choice([4, 4, 8])
    gs = rng.choice([64, 64, 64, 64, 64, 32, 128])
    if kind == "linear":
        K = gs * max(1, _log(rng, 512, 14336) // gs)
        N = _log(rng, 512, 14336)
        M = _log(rng, 1, 2048)
        while M * N * K > 2048 * 14336 * 4096:
            M //= 2
        return {"kind": kind, "M": M, "N": N, "K": K, "bits": bits, "gs": gs}
    if kind == "layers":
        hidden = 128 * rng.randint(8, 32)
        return {"kind": kind, "M": _log(rng, 1, 128), "layers": rng.randint(2, 4), "hidden": hidden, "kv": 128 * rng.randint(2, hidden // 128 // 2),
                "ffn": 128 * _log(rng, 16, 112), "bits": bits, "gs": 64}
    if kind == "attention":
        B, Hkv, T = _log(rng, 1, 16), rng.choice([2, 4, 8]), _log(rng, 64, 32768)
        return {"kind": kind, "B": B, "Hq": Hkv * rng.randint(1, 8), "Hkv": Hkv, "D": rng.choice([64, 128, 128]), "T": T,
                "Tq": rng.choice([1, 1, 1, rng.randint(2, 8)]), "bits": bits, "gs": 64}
    if kind == "tick":
        Hkv, gqa = rng.choice([4, 8]), rng.randint(2, 4)
        return {"kind": kind, "N": _log(rng, 1, 32), "T": _log(rng, 128, 4096), "hidden": 256 * rng.randint(8, 16), "Hq": Hkv * gqa, "Hkv": Hkv,
                "ffn": 256 * rng.randint(16, 56), "bits": bits, "gs": 64}
    if kind == "moe":
        E = rng.choice([32, 64, 128])
        return {"kind": kind, "T": _log(rng, 1, 4096), "E": E, "topk": rng.choice([2, 4, 8]), "H": 256 * rng.randint(4, 8), "I": 128 * rng.randint(4, 12),
                "bits": bits, "gs": 64}
    return {"kind": kind, "B": rng.randint(1, 4), "Hkv": rng.choice([2, 4, 8]), "D": rng.choice([64, 128]), "S": _log(rng, 1, 4096),
            "offset": rng.randint(0, 300), "bits": bits, "gs": 64}


class _Make:
    """Seeded inputs on the GPU: weights ~N(0, 0.02) quantized with the library, activations ~N(0, 1)."""

    def __init__(self, seed, case):
        self.g = torch.Generator(device="cuda").manual_seed(seed)
        self.bits, self.gs = case["bits"], case["gs"]

    def act(self, *shape):
        return torch.randn(shape, device="cuda", generator=self.g, dtype=BF16)

    def weight(self, *shape):
        return qb200.quantize(self.act(*shape).mul_(0.02), self.gs, self.bits)

    def cache(self, *shape):
        return qb200.quantize(self.act(*shape), self.gs, self.bits)

    def lengths(self, n, T):
        """Ragged: between half of T and T, the first one T itself."""
        r = torch.randint(max(1, T // 2), T + 1, (n,), device="cuda", generator=self.g)
        r[0] = T
        return r.to(torch.int32)


def prepare(case, seed):
    return {"linear": _prep_linear, "layers": _prep_layers, "attention": _prep_attention, "tick": _prep_tick, "moe": _prep_moe,
            "cache": _prep_cache}[case["kind"]](case, _Make(seed, case))


def run(state):
    return state["run"](state)


# ---- one quantized linear: x [M, K] . W [N, K]^T, the result allocated by the call ----
def _prep_linear(c, mk):
    return {"run": _run_linear, "c": c, "x": mk.act(c["M"], c["K"]), "w": mk.weight(c["N"], c["K"])}


def _run_linear(s):
    c = s["c"]
    return qb200.quantized_matmul(s["x"], *s["w"], True, c["gs"], c["bits"])


# ---- the projections of decoder layers at a fixed batch, as one CUDA graph ----
def _widths(c):
    h, kv, f = c["hidden"], c["kv"], c["ffn"]
    return [(h, h), (kv, h), (kv, h), (h, h), (f, h), (f, h), (h, f)]   # q k v o gate up down: (out, in)


def _prep_layers(c, mk):
    M, L, wd = c["M"], c["layers"], _widths(c)
    ws = [[mk.weight(n, k) for n, k in wd] for _ in range(L)]
    xh, xf = mk.act(L, M, c["hidden"]), mk.act(L, M, c["ffn"])
    ys = [[torch.empty((M, n), dtype=BF16, device="cuda") for n, _ in wd] for _ in range(L)]
    bits, gs = c["bits"], c["gs"]

    def step():
        for w, y, h, f in zip(ws, ys, xh, xf):
            qb200.quantized_matmul_batch(h, w[0:3], y[0:3], True, gs, bits)
            qb200.quantized_matmul(h, *w[3], True, gs, bits, out=y[3])
            qb200.quantized_matmul_batch(h, w[4:6], y[4:6], True, gs, bits)
            qb200.quantized_matmul(f, *w[6], True, gs, bits, out=y[6])

    step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    return {"run": _run_layers, "graph": graph, "keep": (ws, xh, xf), "ys": ys}


def _run_layers(s):
    s["graph"].replay()
    return s["ys"]


# ---- decode / verify attention over a batch's packed cache (views of larger capacity buffers) ----
def _prep_attention(c, mk):
    B, Hq, Hkv, D, T, Tq = (c[k] for k in ("B", "Hq", "Hkv", "D", "T", "Tq"))
    cap = T + 256
    k = [t[:, :, :T] for t in mk.cache(B, Hkv, cap, D)]
    v = [t[:, :, :T] for t in mk.cache(B, Hkv, cap, D)]
    q = mk.act(B, Hq, Tq, D)
    lens = mk.lengths(B, T) if Tq == 1 else None
    ws = torch.empty(max(16, qb200.kv_decode_attention_workspace_size(B if Tq == 1 else Tq, Hq, Hkv, T, D)), dtype=torch.uint8, device="cuda")
    return {"run": _run_attention, "c": c, "q": q, "k": k, "v": v, "lens": lens, "ws": ws}


def _run_attention(s):
    c = s["c"]
    return qb200.kv_decode_attention(s["q"], s["k"], s["v"], c["bits"], c["gs"], c["D"] ** -0.5, "causal" if c["Tq"] > 1 else "",
                                     kv_lens=s["lens"], workspace=s["ws"])


# ---- one layer of a continuous-batching decode tick ----
def _prep_tick(c, mk):
    N, T, hd, Hq, Hkv, f, D = c["N"], c["T"], c["hidden"], c["Hq"], c["Hkv"], c["ffn"], 128
    w = {n: mk.weight(*s) for n, s in (("q", (Hq * D, hd)), ("k", (Hkv * D, hd)), ("v", (Hkv * D, hd)), ("o", (hd, Hq * D)), ("g", (f, hd)),
                                       ("u", (f, hd)), ("d", (hd, f)))}
    kc, vc = mk.cache(N, Hkv, T + 256, D), mk.cache(N, Hkv, T + 256, D)
    lens = mk.lengths(N, T).tolist()
    seqs = [[t[n:n + 1] for t in c3] for c3 in (kc, vc) for n in range(N)]
    views = [[t[n:n + 1, :, :lens[n]] for t in c3] for c3 in (kc, vc) for n in range(N)]
    qkv = torch.empty((N, (Hq + 2 * Hkv) * D), dtype=BF16, device="cuda")
    new = lambda n: torch.empty((N, n), dtype=BF16, device="cuda")  # noqa: E731
    qb200.swiglu(new(f).zero_(), new(f).zero_())   # the sigmoid table goes up with the first call
    return {"run": _run_tick, "c": c, "w": w, "x": mk.act(N, hd), "n1": (1 + 0.1 * mk.act(hd)).to(BF16), "n2": (1 + 0.1 * mk.act(hd)).to(BF16),
            "cache": (kc, vc), "kt": seqs[:N], "vt": seqs[N:], "kv": views[:N], "vv": views[N:], "pos": [t - 1 for t in lens],
            "outs": [qkv[:, :Hq * D], qkv[:, Hq * D:(Hq + Hkv) * D], qkv[:, (Hq + Hkv) * D:]], "gu": [new(f), new(f)]}


def _run_tick(s):
    c, w, D = s["c"], s["w"], 128
    N, Hq, Hkv, gs, bits = c["N"], c["Hq"], c["Hkv"], c["gs"], c["bits"]
    h = qb200.rms_norm(s["x"], s["n1"], 1e-5)
    q, k, v = qb200.quantized_matmul_batch(h, [w["q"], w["k"], w["v"]], s["outs"], True, gs, bits)
    q = q.view(N, Hq, 1, D)
    qb200.kv_append_seqs(s["kt"], s["vt"], k.view(N, Hkv, 1, D), v.view(N, Hkv, 1, D), s["pos"], bits, gs, rope_q=q, rope_dims=D, rope_base=500000.0)
    a = qb200.kv_decode_attention_ptrs(q, s["kv"], s["vv"], bits, gs, D ** -0.5)
    o = qb200.quantized_matmul(a.view(N, Hq * D), *w["o"], True, gs, bits)
    h1, h = qb200.add_rms_norm(s["x"], o, s["n2"], 1e-5)
    g, u = qb200.quantized_matmul_batch(h, [w["g"], w["u"]], s["gu"], True, gs, bits)
    d = qb200.quantized_matmul(qb200.swiglu(g, u), *w["d"], True, gs, bits)
    h2, h = qb200.add_rms_norm(h1, d, s["n1"], 1e-5)
    return {"residual": h2, "next": h, "k": s["cache"][0], "v": s["cache"][1]}


# ---- the routed-expert block ----
def _prep_moe(c, mk):
    T, E, k, H, inter = c["T"], c["E"], c["topk"], c["H"], c["I"]
    s = {"run": _run_moe_few if T <= 4 else _run_moe, "c": c, "x": mk.act(T, 1, H), "logits": mk.act(T, E).float(), "gate": mk.weight(E, inter, H),
         "up": mk.weight(E, inter, H), "down": mk.weight(E, H, inter), "fused": True}
    try:
        s["run"](s)
    except qb200.Qb200Error:   # a shape the fused entries decline: the host falls through to the separate operators
        s["run"], s["fused"] = _run_moe, False
    return s


def _run_moe_few(s):
    """A few tokens: every (token, slot) by itself, no sort."""
    c = s["c"]
    gs, bits = c["gs"], c["bits"]
    inds, scores = qb200.moe_route(s["logits"], c["topk"])
    scores = scores.to(BF16)
    act = qb200.gather_qmm_swiglu(s["x"].unsqueeze(1), *s["gate"], *s["up"], None, inds, gs, bits)
    y = qb200.moe_down_reduce(act, *s["down"], inds, scores, gs, bits)
    return {"y": y, "experts": inds, "scores": scores}


def _run_moe(s):
    c = s["c"]
    gs, bits = c["gs"], c["bits"]
    inds, scores = qb200.moe_route(s["logits"], c["topk"])
    scores = scores.to(BF16)
    order, inv, sinds, rows, _ = qb200.moe_sort_by_expert(inds, c["E"])
    x = torch.index_select(s["x"], 0, rows)
    if s["fused"]:
        try:
            act = qb200.gather_qmm_swiglu(x, *s["gate"], *s["up"], None, sinds, gs, bits, sorted_indices=True)
        except qb200.Qb200Error:
            s["fused"] = False
    if not s["fused"]:
        g = qb200.gather_qmm(x, *s["gate"], None, sinds, True, gs, bits, sorted_indices=True)
        u = qb200.gather_qmm(x, *s["up"], None, sinds, True, gs, bits, sorted_indices=True)
        act = qb200.swiglu(g, u)
    y = qb200.gather_qmm(act, *s["down"], None, sinds, True, gs, bits, sorted_indices=True)
    return {"y": qb200.moe_weighted_sum(y, scores, inv), "experts": inds, "scores": scores}


# ---- a prompt's keys and values into the packed cache, and the whole of it back as bf16 ----
def _prep_cache(c, mk):
    B, Hkv, D, S, off = (c[k] for k in ("B", "Hkv", "D", "S", "offset"))
    cap = off + S + 256
    return {"run": _run_cache, "c": c, "dense": [mk.act(B, Hkv, S, D) for _ in range(2)], "caches": [mk.cache(B, Hkv, cap, D) for _ in range(2)]}


def _run_cache(s):
    c, out = s["c"], []
    n = c["offset"] + c["S"]
    for dense, (q, sc, bi) in zip(s["dense"], s["caches"]):
        qb200.kv_append(q, sc, bi, dense, c["offset"], c["bits"], c["gs"])
        out.append(qb200.dequantize(q[:, :, :n], sc[:, :, :n], bi[:, :, :n], c["gs"], c["bits"]))
    return {"dense": out, "caches": s["caches"]}


# ---- what a pass cannot do without ----
def _wbytes(n, k, c):
    return n * k * c["bits"] / 8 + 4 * n * k / c["gs"]


def work(case):
    c = case
    if c["kind"] == "linear":
        M, N, K = c["M"], c["N"], c["K"]
        return {"bytes": _wbytes(N, K, c) + 2 * M * (N + K), "flops": 2.0 * M * N * K}
    if c["kind"] == "layers":
        M, L = c["M"], c["layers"]
        wd = _widths(c)
        return {"bytes": L * (sum(_wbytes(n, k, c) + 2 * M * n for n, k in wd) + 2 * M * (c["hidden"] + c["ffn"])),
                "flops": L * 2.0 * M * sum(n * k for n, k in wd)}
    if c["kind"] == "attention":
        tokens = c["B"] * c["T"] * (1.0 if c["Tq"] > 1 or c["B"] == 1 else 0.75 + 0.25 / c["B"])   # lengths between T / 2 and T
        return {"bytes": 2 * _wbytes(tokens * c["Hkv"], c["D"], c) + 4 * c["B"] * c["Hq"] * c["Tq"] * c["D"],
                "flops": 4.0 * tokens * c["Hq"] * c["Tq"] * c["D"]}
    if c["kind"] == "tick":
        N, hd, f, D = c["N"], c["hidden"], c["ffn"], 128
        tokens = N * c["T"] * (1.0 if N == 1 else 0.75 + 0.25 / N)
        w = (2 * c["Hq"] + 2 * c["Hkv"]) * D * hd + 3 * hd * f
        return {"bytes": _wbytes(1, w, c) + 2 * _wbytes(tokens * c["Hkv"], D, c) + 2 * N * 3 * hd,
                "flops": 2.0 * N * w + 4.0 * tokens * c["Hq"] * D}
    if c["kind"] == "moe":
        T, E, k, H, inter = c["T"], c["E"], c["topk"], c["H"], c["I"]
        hit = E * (1 - (1 - k / E) ** T)
        return {"bytes": hit * 3 * _wbytes(inter, H, c) + 4 * T * H + 4 * T * E + 6 * T * k, "flops": 2.0 * T * k * 3 * H * inter}
    B, Hkv, D, S, off = (c[k] for k in ("B", "Hkv", "D", "S", "offset"))
    dense, packed = 2 * B * Hkv * D, _wbytes(B * Hkv, D, c)
    return {"bytes": 2 * (S * (dense + packed) + off * packed + (S + off) * dense), "flops": 0}


def tolerance(case):
    k = case["kind"]
    if k == "cache":
        return "exact"             # codes, scales, biases and the dequantized values are defined to the bit
    if k in ("linear", "layers"):
        return {"rel": 5e-3, "max": 3e-2}   # one bf16 rounding of the result (and of the weight at wide batches)
    if k == "attention":
        return {"rel": 1e-2, "max": 1e-1}
    # chains of bf16 results; a code of a new cache row may fall on the other side of a rounding boundary
    return {"rel": 1e-2, "max": 2e-1, "differ": 2e-3}
