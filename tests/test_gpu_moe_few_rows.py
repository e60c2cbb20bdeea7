"""The MoE layer at few rows per expert, on either side of each line of the weight-streaming kernel's dispatch: one, two or
four token tiles of eight, experts with more rows than an item holds, K split over a CTA's warps or not (with the
quantisation in a kernel of its own), one and two activation terms, routing and placement in one kernel (up to 32 tokens)
or two, and the tcgen05 core just beyond.  Oracle and tolerance of test_gpu_moe.py's layer test."""
import functools

import pytest
import torch

import open_cake_ir_b200 as cake
from oracle import compare, moe as oracle_moe, routing as oracle_routing
from test_gpu_moe import run_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,hidden,inter,experts,local,offset,act", [
    (1, 1024, 256, 64, 64, 0, "split"), (3, 512, 128, 64, 16, 32, "fp8"), (20, 1024, 256, 64, 64, 0, "fp8"),      # one token tile
    (30, 1024, 512, 64, 64, 0, "split"), (32, 2048, 256, 32, 8, 8, "fp8"), (33, 1024, 256, 32, 32, 0, "split"),   # two
    (42, 1024, 256, 32, 32, 0, "split"), (44, 256, 384, 32, 4, 28, "fp8"), (45, 256, 384, 32, 4, 28, "fp8"),      # four; the core
    (60, 512, 512, 64, 64, 0, "fp8"), (61, 512, 512, 64, 64, 0, "split")])        # more tiles than SMs: two; the core
def test_few_rows_per_expert(tokens, hidden, inter, experts, local, offset, act):
    cpu = cake.workloads.moe_inputs(tokens, hidden, inter, experts, local, offset, routing="softmax", device="cpu")
    # every token goes to one expert of this rank, which so has more rows than an item or a tile holds
    cpu["routing_logits"][:, offset] += 8.0
    out, _ = run_layer(cpu, experts=experts, routing="softmax", act_mode=act)
    want = oracle_moe.moe_reference(cpu, routing="softmax", act_quant="fp8" if act == "fp8" else "none", dtype=torch.float32)
    assert compare.rel_frobenius(out, want["output"]) <= (1e-2 if act == "fp8" else 4e-3)


@pytest.mark.parametrize("act", ["fp8", "split"])
@pytest.mark.parametrize("tokens", [12, 200])          # the weight-streaming kernel; the tcgen05 core, tiles of 128 and 72 rows
def test_gates_at_the_ends_of_the_sigmoid(tokens, act):
    """Gates of several hundred either way: the sigmoid is 0 or 1 to the last bit, and nothing overflows on the way there."""
    experts, offset = 8, 0
    cpu = cake.workloads.moe_inputs(tokens, 512, 256, experts, experts, offset, routing="softmax", device="cpu")
    cpu["gemm1_weights_scale"] = cpu["gemm1_weights_scale"] * 300
    out, _ = run_layer(cpu, experts=experts, routing="softmax", act_mode=act)
    want = oracle_moe.moe_reference(cpu, routing="softmax", act_quant="fp8" if act == "fp8" else "none", dtype=torch.float32)
    assert torch.isfinite(out.float()).all()
    assert compare.rel_frobenius(out, want["output"]) <= (1e-2 if act == "fp8" else 4e-3)


@functools.lru_cache(maxsize=1)
def large_experts():
    """16 of 64 experts, large enough that streaming one several times costs more than the core's launches."""
    return cake.workloads.moe_inputs(56, 4096, 2304, 64, 16, 0, routing="softmax", device="cpu")


@pytest.mark.parametrize("act", ["fp8", "split"])
@pytest.mark.parametrize("tokens,equal,offset", [
    (24, 17, 0), (24, 16, 0),         # one row above the line and on it; up to 32 tokens
    (24, 20, 5),                      # three of the experts of many rows are this rank's: not worth the core's launches
    (56, 56, 0),                      # every row is the core's
    (56, 29, 0), (56, 28, 0)])        # both kernels have experts; on the line
def test_uneven_routing(tokens, equal, offset, act):
    """Tokens that all go to the same experts, as a batch of one prompt or the padding of one does, among others: on either side
    of each line that sends experts of many rows to the tcgen05 core."""
    cpu = dict(large_experts(), local_expert_offset=torch.tensor([offset], dtype=torch.int32))
    for name in ("routing_logits", "hidden_states"):
        cpu[name] = cpu[name][:tokens].clone()
    cpu["hidden_states_scale"] = cpu["hidden_states_scale"][:, :tokens].contiguous()
    cpu["routing_logits"][:equal, :8] += 20.0
    cpu["routing_logits"][equal:, :8] -= 20.0
    out, _ = run_layer(cpu, experts=64, routing="softmax", act_mode=act)
    want = oracle_moe.moe_reference(cpu, routing="softmax", act_quant="fp8" if act == "fp8" else "none", dtype=torch.float32)
    assert compare.rel_frobenius(out, want["output"]) <= (1e-2 if act == "fp8" else 4e-3)


@pytest.mark.parametrize("tokens,hidden,inter,experts,local,offset,act", [
    (5, 1024, 256, 64, 16, 16, "fp8"),           # K split over warps, quantisation in a kernel of its own
    (40, 512, 256, 64, 64, 0, "split"),          # one warp to a sub-tile; no pairs of other ranks
    (40, 512, 256, 64, 16, 32, "fp8")])
def test_external_routing_at_few_rows(tokens, hidden, inter, experts, local, offset, act):
    """Selections and weights from outside, as an expert-parallel step hands them over: some of other ranks, some rows absent (-1)."""
    cpu = cake.workloads.moe_inputs(tokens, hidden, inter, experts, local, offset, routing="softmax", device="cpu")
    ids, weights = oracle_routing.routing_softmax_topk(cpu["routing_logits"])
    ids, weights = ids.int(), weights.float() * 2.5
    absent = torch.arange(tokens) % 5 == 4
    ids[absent] = -1
    inputs = {k: v for k, v in cpu.items() if k not in ("routing_logits", "routing_bias")}
    out, _ = run_layer(dict(inputs, expert_ids=ids, route_weights=weights), experts=experts, act_mode=act, external_routing=True)
    want = oracle_moe.moe_reference(dict(cpu, routed_scaling_factor=torch.tensor([2.5])), routing="softmax", act_quant="fp8" if act == "fp8" else "none",
                                    dtype=torch.float32)["output"]
    assert not bool(out[absent.cuda()].any())
    assert compare.rel_frobenius(out[~absent.cuda()], want[~absent]) <= (1e-2 if act == "fp8" else 4e-3)
