"""The work that is timed when this library's speed is looked at: calls through the public operator objects, as a
serving program makes them.  Such a program builds an operator object once over its buffers (weights, KV cache,
activations, outputs, workspace) and calls ``launch`` each step on the current stream; that launch is what a pass is.

    listed()              the named cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   buffers and operator object, on the GPU
    run(state)            one launch; returns the outputs
    work(case)            bytes and floating-point operations of a pass that no implementation can avoid
    tolerance(case)       how far two correct implementations at the same precision may be apart

Sizes are those of the workloads of this repository (``bench.py``, ``open_cake_ir_b200.workloads``, ``tests/``) and,
around them, what a server meets: steps of one token up to whole prompts, one rank's share of the experts up to all
of them, short and long sequences, small and large pages, few and many heads.
"""
from __future__ import annotations

import math

import torch

import open_cake_ir_b200 as cake

BF16, E4M3, F32, I32 = torch.bfloat16, torch.float8_e4m3fn, torch.float32, torch.int32


# ------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # The norms of a decode step: a few dozen rows, residual added and handed on.  Latency and launch cost.
        {"name": "add_rmsnorm_decode", "op": "norm", "form": "add", "rows": 64, "width": 7168},
        # The norm of a prefill step (and the RMSNorm workload of the benchmark).
        {"name": "rmsnorm_prefill", "op": "norm", "form": "plain", "rows": 4096, "width": 4096},
        # A projection in a decode step: few rows against a whole weight matrix, so the weights have to stream.
        {"name": "gemm_decode", "op": "gemm", "m": 64, "n": 4096, "k": 7168},
        # The same projection in a prefill step (the GEMM workload of the benchmark): bound by the tensor cores.
        {"name": "gemm_prefill", "op": "gemm", "m": 8192, "n": 4096, "k": 7168},
        # One token on a rank that holds an eighth of the experts, in the mode that meets the reference contract's
        # tolerance (its MoE cases are this shape): about one routed pair, so launches and latency.
        {"name": "moe_one_token", "op": "moe", "tokens": 1, "hidden": 7168, "inter": 2048, "experts": 256, "local": 32,
         "routing": "ds", "act": "split"},
        # A decode step of 64 sequences over all experts on one GPU: nearly every expert's weights for two rows each.
        {"name": "moe_decode", "op": "moe", "tokens": 64, "hidden": 7168, "inter": 2048, "experts": 256, "local": 256,
         "routing": "ds", "act": "fp8"},
        # The MoE workload of the benchmark: 4096 tokens, 128 per expert.
        {"name": "moe_prefill", "op": "moe", "tokens": 4096, "hidden": 7168, "inter": 2048, "experts": 256, "local": 256,
         "routing": "softmax", "act": "fp8"},
        # A decode step of a full batch (the GQA workload of the benchmark): bound by the KV stream.
        {"name": "gqa_decode_batch", "op": "gqa_decode", "batch": 64, "hq": 32, "hkv": 8, "page": 16, "lo": 512, "hi": 4096},
        # A decode step of a few long conversations: little work per step, cut over the whole GPU and merged.
        {"name": "gqa_decode_long", "op": "gqa_decode", "batch": 3, "hq": 32, "hkv": 8, "page": 16, "lo": 9000, "hi": 32768},
        # The MLA workload of the benchmark: 128 heads over one latent row per token.
        {"name": "mla_decode_batch", "op": "mla_decode", "batch": 32, "heads": 128, "page": 64, "lo": 1024, "hi": 8192},
        # Prompts of a chat server, one of them continuing after a cached prefix, over the paged cache.
        {"name": "gqa_prefill_paged", "op": "gqa_prefill", "segments": 4, "new": 8000, "prefix": 1000, "hq": 32, "hkv": 8,
         "page": 16, "paged": True},
        # A chunk of prompts over the paged latent cache, behind what earlier chunks have left there.
        {"name": "mla_prefill_paged", "op": "mla_prefill", "segments": 2, "new": 1500, "prefix": 700, "heads": 128, "page": 64},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _whole(rng, lo, hi, multiple=1):
    """A size whose logarithm is spread evenly over [lo, hi], rounded to a multiple."""
    return max(lo, min(hi, int(round(_log(rng, lo, hi) / multiple)) * multiple))


def draw(rng):
    # operators as often as they are listed
    op = rng.choice(["norm", "norm", "gemm", "gemm", "moe", "moe", "moe", "gqa_decode", "gqa_decode", "mla_decode",
                     "gqa_prefill", "mla_prefill"])
    if op == "norm":
        width = rng.choice([512, 1536, 2048, 4096, 7168, 8192, _whole(rng, 256, 16384, 8)])
        return {"op": op, "form": rng.choice(["plain", "residual", "add"]), "rows": _whole(rng, 1, 8192), "width": width}
    if op == "gemm":
        return {"op": op, "m": _whole(rng, 1, 8192), "n": _whole(rng, 512, 8192, 128), "k": _whole(rng, 512, 7168, 128)}
    if op == "moe":
        hidden, inter, experts, local = rng.choice([(7168, 2048, 256, 32), (7168, 2048, 256, 64), (7168, 2048, 256, 128),
                                                    (7168, 2048, 256, 256), (2048, 768, 128, 128), (4096, 1536, 128, 32),
                                                    (1024, 512, 64, 64)])
        return {"op": op, "tokens": _whole(rng, 1, 4096), "hidden": hidden, "inter": inter, "experts": experts, "local": local,
                "routing": rng.choice(["ds", "softmax"]), "act": rng.choice(["fp8", "fp8", "split"])}
    if op == "gqa_decode":
        hq, hkv = rng.choice([(32, 8), (32, 8), (64, 8), (32, 4), (16, 2), (8, 8), (24, 3), (64, 16), (8, 1)])
        hi = _whole(rng, 256, 32768)
        batch = _whole(rng, 1, max(1, min(128, 300000 // hi)))
        return {"op": op, "batch": batch, "hq": hq, "hkv": hkv, "page": rng.choice([1, 16, 16, 64]), "lo": max(1, hi // rng.choice([2, 4, 8])), "hi": hi}
    if op == "mla_decode":
        hi = _whole(rng, 256, 32768)
        batch = _whole(rng, 1, max(1, min(128, 300000 // hi)))
        return {"op": op, "batch": batch, "heads": rng.choice([16, 32, 64, 128, 128]), "page": rng.choice([1, 16, 64, 64]),
                "lo": max(1, hi // rng.choice([2, 4, 8])), "hi": hi}
    segments = _whole(rng, 1, 8)
    if op == "gqa_prefill":
        hq, hkv = rng.choice([(32, 8), (32, 8), (64, 8), (32, 4), (16, 2), (8, 8), (24, 3), (40, 8)])
        case = {"op": op, "segments": segments, "new": _whole(rng, 16 * segments, 6000), "prefix": rng.choice([0, 0, _whole(rng, 16, 2000)]),
                "hq": hq, "hkv": hkv, "page": rng.choice([1, 16, 16, 64]), "paged": rng.choice([True, True, False])}
    else:
        case = {"op": op, "segments": segments, "new": _whole(rng, 16 * segments, 1500), "prefix": rng.choice([0, 0, _whole(rng, 16, 700)]),
                "heads": rng.choice([16, 32, 64, 128, 128]), "page": rng.choice([1, 16, 64, 64])}
    largest = next(c for c in listed() if c["op"] == op)
    while _visible_pairs(case) * case.get("hkv", 1) > _visible_pairs(largest) * largest.get("hkv", 1):      # no more than what is listed
        case["new"] = max(segments, case["new"] * 3 // 4)
    return case


# ----------------------------------------------------------------------------------------- inputs
def _spread(count, lo, hi):
    """``count`` lengths spread evenly over [lo, hi]; the same for every seed, so that the work of a case is fixed."""
    if count == 1:
        return [(lo + hi) // 2 | 1]
    return [lo + (hi - lo) * i // (count - 1) for i in range(count)]


def _split(total, parts):
    """``total`` cut into ``parts`` uneven pieces of at least one."""
    shares = [2 + i for i in range(parts)]
    out = [max(1, total * s // sum(shares)) for s in shares]
    out[-1] += total - sum(out)
    return out


def _decode_lengths(case):
    return _spread(case["batch"], case["lo"], case["hi"])


def _prefill_lengths(case):
    """(new rows, KV rows) of each segment; every second segment continues behind a cached prefix."""
    new = _split(case["new"], case["segments"])
    return new, [n + (case["prefix"] if i % 2 == 0 else 0) for i, n in enumerate(new)]


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device="cuda", dtype=F32)


def _bf16(g, *shape):
    return torch.randn(shape, generator=g, device="cuda", dtype=BF16)


def _order(g, lengths):
    """The lengths in an order that the seed decides."""
    return [lengths[i] for i in torch.randperm(len(lengths), generator=g, device="cuda").tolist()]


def _prefix_sum(values):
    out = [0]
    for v in values:
        out.append(out[-1] + v)
    return torch.tensor(out, dtype=I32, device="cuda")


def _pages(g, lengths, page):
    """Page table of sequences of these lengths: pages are entries of a permutation of a pool a little larger than needed."""
    counts = [(n + page - 1) // page for n in lengths]
    pool = sum(counts) + 64
    indices = torch.randperm(pool, generator=g, device="cuda")[:sum(counts)].to(I32)
    last = torch.tensor([n - (c - 1) * page if c else 0 for n, c in zip(lengths, counts)], dtype=I32, device="cuda")
    return pool, _prefix_sum(counts), indices, last


def _scale(value):
    return torch.tensor([value], dtype=F32, device="cuda")


def _quantized_rows(g, rows, k):
    return cake.workloads.quantize_rows_1x128(_randn(g, rows, k))


def _quantized_blocks(g, n, k, std=1.0):
    return cake.workloads.quantize_blocks_128x128(_randn(g, n, k) * std)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    return _PREPARE[case["op"]](case, g)


def _prepare_norm(case, g):
    rows, width = case["rows"], case["width"]
    x, weight = _bf16(g, rows, width), (1 + 0.1 * _randn(g, width)).to(BF16)
    out = torch.empty_like(x)
    if case["form"] == "plain":
        return {"op": cake.RmsNorm(x, weight, out, 1e-6), "outputs": [out]}
    residual = _bf16(g, rows, width)
    if case["form"] == "residual":
        return {"op": cake.RmsNorm(x, weight, out, 1e-6, residual), "outputs": [out]}
    residual_out = torch.empty_like(x)
    return {"op": cake.AddRmsNorm(x, residual, weight, out, residual_out, 1e-6), "outputs": [out, residual_out]}


def _prepare_gemm(case, g):
    a, sfa = _quantized_rows(g, case["m"], case["k"])
    b, sfb = _quantized_blocks(g, case["n"], case["k"])
    c = torch.empty((case["m"], case["n"]), dtype=BF16, device="cuda")
    return {"op": cake.BlockScaledGemm(a, sfa, b, sfb, c), "outputs": [c]}


def _prepare_moe(case, g):
    tokens, hidden, inter, experts, local = (case[k] for k in ("tokens", "hidden", "inter", "experts", "local"))
    h, hs = _quantized_rows(g, tokens, hidden)
    w13 = torch.empty((local, 2 * inter, hidden), dtype=E4M3, device="cuda")
    s13 = torch.empty((local, 2 * inter // 128, hidden // 128), dtype=F32, device="cuda")
    w2 = torch.empty((local, hidden, inter), dtype=E4M3, device="cuda")
    s2 = torch.empty((local, hidden // 128, inter // 128), dtype=F32, device="cuda")
    for e in range(local):
        w13[e], s13[e] = _quantized_blocks(g, 2 * inter, hidden, hidden ** -0.5)
        w2[e], s2[e] = _quantized_blocks(g, hidden, inter, inter ** -0.5)
    bias = torch.zeros(experts, dtype=BF16, device="cuda")
    if case["routing"] == "ds":
        bias = (torch.rand(experts, generator=g, device="cuda") * 0.015).to(BF16)
    ranks = experts // local
    first = local * int(torch.randint(ranks, (1,), generator=g, device="cuda"))      # this rank's share of the experts
    logits = _randn(g, tokens, experts)
    if tokens * 8 < 4 * ranks:      # a step of very few tokens reaches this rank because it holds one of their experts
        logits[0, first + int(torch.randint(local, (1,), generator=g, device="cuda"))] = 6.0
    inputs = {"routing_logits": logits, "routing_bias": bias, "hidden_states": h, "hidden_states_scale": hs,
              "gemm1_weights": w13, "gemm1_weights_scale": s13, "gemm2_weights": w2, "gemm2_weights_scale": s2,
              "local_expert_offset": torch.tensor([first], dtype=I32, device="cuda"), "routed_scaling_factor": _scale(2.5)}
    output = torch.empty((tokens, hidden), dtype=BF16, device="cuda")
    return {"op": cake.Fp8Moe(inputs, output, experts=experts, routing=case["routing"], act_mode=case["act"]), "outputs": [output]}


def _prepare_gqa_decode(case, g):
    lengths = _order(g, _decode_lengths(case))
    batch, hq, hkv, page = case["batch"], case["hq"], case["hkv"], case["page"]
    pool, indptr, indices, last = _pages(g, lengths, page)
    q, k, v = _bf16(g, batch, hq, 128), _bf16(g, pool, page, hkv, 128), _bf16(g, pool, page, hkv, 128)
    output, lse = torch.empty_like(q), torch.empty((batch, hq), dtype=F32, device="cuda")
    return {"op": cake.GqaPagedDecode(q, k, v, indptr, indices, last, _scale(128 ** -0.5), output, lse, max_kv_len=case["hi"]),
            "outputs": [output, lse]}


def _prepare_mla_decode(case, g):
    lengths = _order(g, _decode_lengths(case))
    batch, heads, page = case["batch"], case["heads"], case["page"]
    pool, indptr, indices, last = _pages(g, lengths, page)
    q_nope, q_pe = _bf16(g, batch, heads, 512), _bf16(g, batch, heads, 64)
    ckv, kpe = _bf16(g, pool, page, 512), _bf16(g, pool, page, 64)
    output, lse = torch.empty_like(q_nope), torch.empty((batch, heads), dtype=F32, device="cuda")
    return {"op": cake.MlaPagedDecode(q_nope, q_pe, ckv, kpe, indptr, indices, last, _scale(192 ** -0.5), output, lse,
                                      max_kv_len=case["hi"]), "outputs": [output, lse]}


def _prepare_gqa_prefill(case, g):
    new, kv = _prefill_lengths(case)
    total, hq, hkv, page = sum(new), case["hq"], case["hkv"], case["page"]
    q = _bf16(g, total, hq, 128)
    output, lse = torch.empty_like(q), torch.empty((total, hq), dtype=F32, device="cuda")
    if case["paged"]:
        pool, indptr, indices, last = _pages(g, kv, page)
        k, v = _bf16(g, pool, page, hkv, 128), _bf16(g, pool, page, hkv, 128)
    else:
        indptr, indices, last = _prefix_sum(kv), None, None
        k, v = _bf16(g, sum(kv), hkv, 128), _bf16(g, sum(kv), hkv, 128)
    return {"op": cake.GqaCausalPrefill(q, k, v, _prefix_sum(new), indptr, indices, last, _scale(128 ** -0.5), output, lse,
                                        max_kv_len=max(kv)), "outputs": [output, lse]}


def _prepare_mla_prefill(case, g):
    new, kv = _prefill_lengths(case)
    total, heads, page = sum(new), case["heads"], case["page"]
    pool, indptr, indices, last = _pages(g, kv, page)
    q_nope, q_pe = _bf16(g, total, heads, 512), _bf16(g, total, heads, 64)
    ckv, kpe = _bf16(g, pool, page, 512), _bf16(g, pool, page, 64)
    output, lse = torch.empty_like(q_nope), torch.empty((total, heads), dtype=F32, device="cuda")
    return {"op": cake.MlaCausalPrefill(q_nope, q_pe, ckv, kpe, _prefix_sum(new), indptr, indices, last, _scale(192 ** -0.5), output,
                                        lse, max_kv_len=max(kv)), "outputs": [output, lse]}


_PREPARE = {"norm": _prepare_norm, "gemm": _prepare_gemm, "moe": _prepare_moe, "gqa_decode": _prepare_gqa_decode,
            "mla_decode": _prepare_mla_decode, "gqa_prefill": _prepare_gqa_prefill, "mla_prefill": _prepare_mla_prefill}


def run(state):
    state["op"].launch()
    return state["outputs"]


# ------------------------------------------------------------------------------ work and tolerance
def _visible_pairs(case):
    """(query row, visible KV row) pairs of a causal prefill."""
    return sum(n * (kv - n) + n * (n + 1) // 2 for n, kv in zip(*_prefill_lengths(case)))


def work(case):
    op = case["op"]
    if op == "norm":
        tensors = {"plain": 2, "residual": 3, "add": 4}[case["form"]]
        return {"bytes": 2 * case["width"] * (tensors * case["rows"] + 1), "flops": 4 * case["rows"] * case["width"]}
    if op == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        scales = 4 * (k // 128) * (m + n // 128)
        return {"bytes": m * k + n * k + scales + 2 * m * n, "flops": 2 * m * n * k}
    if op == "moe":
        tokens, hidden, inter, experts, local = (case[k] for k in ("tokens", "hidden", "inter", "experts", "local"))
        pairs = max(1.0, tokens * 8 * local / experts)                         # routed to this rank, on average
        touched = max(1.0, local * (1 - (1 - 8 / experts) ** tokens))          # its experts that get a token, on average
        weights = touched * 3 * inter * hidden * (1 + 4 / 16384)
        rows = tokens * (hidden + 4 * hidden // 128 + 4 * experts + 2 * hidden)
        return {"bytes": weights + rows, "flops": pairs * 6 * inter * hidden}
    if op == "gqa_decode":
        tokens, batch, hq, hkv = sum(_decode_lengths(case)), case["batch"], case["hq"], case["hkv"]
        return {"bytes": tokens * hkv * 512 + 4 * tokens // case["page"] + batch * hq * (512 + 4), "flops": tokens * hq * 4 * 128}
    if op == "mla_decode":
        tokens, batch, heads = sum(_decode_lengths(case)), case["batch"], case["heads"]
        return {"bytes": tokens * 1152 + 4 * tokens // case["page"] + batch * heads * (2 * (576 + 512) + 4),
                "flops": tokens * heads * 2 * (576 + 512)}
    new, kv = _prefill_lengths(case)
    if op == "gqa_prefill":
        return {"bytes": sum(kv) * case["hkv"] * 512 + sum(new) * case["hq"] * (512 + 4), "flops": _visible_pairs(case) * case["hq"] * 4 * 128}
    return {"bytes": sum(kv) * 1152 + sum(new) * case["heads"] * (2 * (576 + 512) + 4),
            "flops": _visible_pairs(case) * case["heads"] * 2 * (576 + 512)}


def tolerance(case):
    # bf16 results of fp32 sums: two correct ones differ where the sum lies near a rounding boundary, by one unit of
    # the last place (2^-8 of the value).  The MoE layer also rounds its intermediate to e4m3 and each contribution
    # row to bf16, where a sum in another order may fall on the other side.
    if case["op"] == "moe":
        return {"rel": 1e-2, "max": 0.1}
    return {"rel": 4e-3, "max": 0.04}
