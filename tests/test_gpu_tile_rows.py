"""The grouped GEMMs at the edges of their row tiles: experts of 1 to 182 rows, whose (last) tile is one of 32, 64 or 128 rows, in one
layer, with one and two activation terms and widths of whole and half column tiles.  The dense GEMM's last row tile likewise.
Oracles and tolerances of test_gpu_moe.py's layer test and test_gpu_gemm.py."""
import pytest
import torch

import open_cake_ir_b200 as cake
from oracle import compare, moe as oracle_moe
from test_gpu_gemm import run
from test_gpu_moe import run_layer

pytestmark = pytest.mark.gpu

TOKENS, ROWS = 183, [1, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160, 161, 182]


def selections():
    """Eight experts of 16 for each token, so that expert e is chosen ROWS[e] times: always those with most rows still to give."""
    left, out = list(ROWS), torch.zeros((TOKENS, 16), dtype=torch.bool)
    for t in range(TOKENS):
        for e in sorted(range(16), key=lambda e: -left[e])[:8]:
            out[t, e] = True
            left[e] -= 1
    assert not any(left)
    return out[torch.randperm(TOKENS, generator=torch.Generator().manual_seed(4))]


@pytest.mark.parametrize("act", ["fp8", "split"])
@pytest.mark.parametrize("hidden,inter", [(512, 384), (640, 128), (128, 256)])
def test_rows_of_an_expert(hidden, inter, act):
    cpu = cake.workloads.moe_inputs(TOKENS, hidden, inter, 16, 16, 0, routing="softmax", device="cpu")
    cpu["routing_logits"] = torch.where(selections(), cpu["routing_logits"] + 20.0, cpu["routing_logits"] - 20.0)
    out, _ = run_layer(cpu, experts=16, routing="softmax", act_mode=act)
    want = oracle_moe.moe_reference(cpu, routing="softmax", act_quant="fp8" if act == "fp8" else "none", dtype=torch.float32)
    assert compare.rel_frobenius(out, want["output"]) <= (1e-2 if act == "fp8" else 4e-3)
    rows = torch.linalg.vector_norm(out.cpu().float() - want["output"].float(), dim=1) / torch.linalg.vector_norm(want["output"].float(), dim=1)
    assert float(rows.max()) <= (4e-2 if act == "fp8" else 1.6e-2)      # of one row in 183: four times the whole, as a wrong row would be far beyond


@pytest.mark.parametrize("m", [2048 + 1, 2048 + 32, 2048 + 33, 2048 + 64, 2048 + 65])
@pytest.mark.parametrize("n", [4096, 4224])
def test_last_tile_of_a_dense_product(m, n):
    c, want = run(m, n, 384)
    ok, bad, err = compare.compare(c, want, atol=2e-2, rtol=2e-2)
    assert ok, f"{bad} mismatches, max abs err {err}"
    assert compare.rel_frobenius(c, want) <= 1e-2


@pytest.mark.parametrize("tokens,experts,inter,act", [
    (20, 32, 256, "fp8"), (21, 32, 256, "fp8"),                # five rows an expert; beyond
    (12, 32, 256, "split"), (13, 32, 256, "split"),            # three: an item of 8 rows, of 16
    (16, 128, 256, "fp8"), (20, 128, 256, "fp8"),              # tiles to 148 SMs: 1.1 and 1.26
    (28, 256, 256, "split"), (31, 256, 256, "split")])         # with two terms: 2.04 and 2.17
def test_lines_of_the_dispatch(tokens, experts, inter, act):
    cpu = cake.workloads.moe_inputs(tokens, 512, inter, experts, experts, 0, routing="softmax", device="cpu")
    out, _ = run_layer(cpu, experts=experts, routing="softmax", act_mode=act)
    want = oracle_moe.moe_reference(cpu, routing="softmax", act_quant="fp8" if act == "fp8" else "none", dtype=torch.float32)
    assert compare.rel_frobenius(out, want["output"]) <= (1e-2 if act == "fp8" else 4e-3)
