"""Attention outputs that start 8 or 16 bytes behind a 32-byte boundary, as a view into a larger buffer does: the same bits
as an aligned output, for sequences that are empty, lie in one range of the work list and are cut by it, and for both
forms of the GQA prefill.  What cannot be written eight bytes at a time is refused when the operator is made."""
import pytest
import torch

import open_cake_ir_b200 as cake
from test_gpu_mla_tiles import paged
from test_gpu_prefill_tiles import problem

pytestmark = pytest.mark.gpu


def mla_decode(dev, out, lse):
    return cake.MlaPagedDecode(dev["q_nope"], dev["q_pe"], dev["ckv_cache"], dev["kpe_cache"], dev["kv_indptr"], dev["kv_indices"],
                               dev["kv_last_page_len"], dev["sm_scale"], out, lse, max_kv_len=2500)


def mla_prefill(dev, out, lse):
    return cake.MlaCausalPrefill(dev["q_nope"], dev["q_pe"], dev["ckv_cache"], dev["kpe_cache"], dev["qo_indptr"], dev["kv_indptr"],
                                 dev["kv_indices"], dev["kv_last_page_len"], dev["sm_scale"], out, lse, max_kv_len=600)


def sparse_mla_decode(dev, out, lse):
    return cake.SparseMlaDecode(dev["q_nope"], dev["q_pe"], dev["ckv_cache"], dev["kpe_cache"], dev["sparse_indices"], out)


def gqa_decode(dev, out, lse):
    return cake.GqaPagedDecode(dev["q"], dev["k_cache"], dev["v_cache"], dev["kv_indptr"], dev["kv_indices"], dev["kv_last_page_len"],
                               dev["sm_scale"], out, lse, max_kv_len=3000)


def gqa_prefill(dev, out, lse):
    return cake.GqaCausalPrefill(dev["q"], dev["k_cache"], dev["v_cache"], dev["qo_indptr"], dev["kv_indptr"], dev["kv_indices"],
                                 dev["kv_last_page_len"], dev["sm_scale"], out, lse, max_kv_len=int(dev["max_kv_len"]))


def inputs(name):
    g = torch.Generator().manual_seed(11)
    if name == "mla_prefill":                                # 48 heads: two tokens to a tile; a segment without KV rows
        cpu = paged(g, [2, 0, 600], 16, 48, 9)
        cpu["qo_indptr"] = torch.tensor([0, 5, 7, 9], dtype=torch.int32)
    elif name in ("mla_decode", "sparse_mla_decode"):
        cpu = paged(g, [0, 5, 2500, 64], 16, 16, 4)
        cpu["sparse_indices"] = torch.arange(4 * 700, dtype=torch.int32).reshape(4, 700) % 2500
        cpu["sparse_indices"][1] = -1
    elif name == "gqa_decode":                               # as many query rows as sequences
        cpu = problem(3, [1] * 4, [0, 3, 3000, 40], 8, 2, 16)
    else:                                                    # tiles; a decode sequence per query row
        cpu = problem(4, [70, 3, 0], [130, 0, 9], 8, 2, 16) if name == "gqa_prefill_tiles" else problem(5, [2, 1], [6000, 0], 8, 1, 16)
        cpu["max_kv_len"] = torch.tensor(130 if name == "gqa_prefill_tiles" else 6000)
    return {k: v.cuda() for k, v in cpu.items()}


@pytest.mark.parametrize("name,make", [("mla_decode", mla_decode), ("mla_prefill", mla_prefill), ("sparse_mla_decode", sparse_mla_decode),
                                       ("gqa_decode", gqa_decode), ("gqa_prefill_tiles", gqa_prefill), ("gqa_prefill_rows", gqa_prefill)])
def test_views_into_a_larger_buffer(name, make):
    dev = inputs(name)
    q = dev.get("q_nope", dev.get("q"))
    lse = torch.empty(q.shape[:2], device="cuda")

    def at(offset):
        raw = torch.full((q.numel() * 2 + 128,), 0xA5, dtype=torch.uint8, device="cuda")
        return raw, raw[offset:offset + q.numel() * 2].view(torch.bfloat16).reshape(q.shape)
    _, want = at(0)
    make(dev, want, lse).launch()
    for offset in (8, 16, 40):
        raw, out = at(offset)
        make(dev, out, lse).launch()
        torch.cuda.synchronize()
        assert torch.equal(out.view(torch.int16), want.view(torch.int16)), f"{offset} bytes into the buffer"
        assert bool((raw[:offset] == 0xA5).all()) and bool((raw[offset + q.numel() * 2:] == 0xA5).all())
    for offset in (2, 4):
        with pytest.raises(cake._lib.CakeError):
            make(dev, at(offset)[1], lse)


def test_moe_output_has_to_be_aligned():
    """The rows that combine the experts' contributions are written 16 bytes at a time."""
    dev = {k: v.cuda() for k, v in cake.workloads.moe_inputs(3, 512, 128, 16, 16, routing="softmax", device="cpu").items()}
    raw = torch.zeros(3 * 512 + 8, dtype=torch.bfloat16, device="cuda")
    op = cake.Fp8Moe(dev, raw[4:4 + 3 * 512].reshape(3, 512), experts=16, routing="softmax")
    with pytest.raises(cake._lib.CakeError):
        op.launch()
    torch.cuda.synchronize()
    assert not bool(raw.any())
