"""MLA attention at the sizes where its tiles can go wrong: lengths on either side of a work unit (32 tokens) and a tile
(64), sequences that a range boundary cuts and ones that lie in one range, head counts that leave rows of a cluster
empty or take two, and query tokens packed several to a tile.  Oracle and tolerance of test_gpu_prefill.py."""
import pytest
import torch

from oracle import attention
from test_gpu_decode import check as check_decode, run_mla
from test_gpu_prefill import check, run

pytestmark = pytest.mark.gpu


def paged(g, kv_lens, page, heads, rows):
    kv_lens = torch.tensor(kv_lens)
    pages = (kv_lens + page - 1) // page
    pool = int(pages.sum()) + 3
    zero = torch.zeros(1, dtype=torch.long)
    return {"q_nope": torch.randn((rows, heads, 512), generator=g).to(torch.bfloat16),
            "q_pe": torch.randn((rows, heads, 64), generator=g).to(torch.bfloat16),
            "ckv_cache": torch.randn((pool, page, 512), generator=g).to(torch.bfloat16),
            "kpe_cache": torch.randn((pool, page, 64), generator=g).to(torch.bfloat16),
            "kv_indptr": torch.cat([zero, pages.cumsum(0)]).int(), "kv_indices": torch.randperm(pool, generator=g)[:int(pages.sum())].int(),
            "kv_last_page_len": torch.where(pages > 0, kv_lens - (pages - 1) * page, torch.zeros_like(kv_lens)).int(),
            "sm_scale": torch.tensor([192.0 ** -0.5])}


@pytest.mark.parametrize("lens,heads,page", [
    ([1, 31, 32, 33, 63, 64, 65, 0, 95, 97, 128, 129], 128, 16), ([2500], 65, 1), ([700, 0, 3, 1300], 200, 64),
    ([64] * 90, 1, 64)])
def test_decode_tile_edges(lens, heads, page):
    cpu = paged(torch.Generator().manual_seed(len(lens) + heads), lens, page, heads, len(lens))
    want = attention.paged_decode_reference(cpu, mla=True, page_size=page, per_head_loop=False)
    out, lse = run_mla(cpu, max(lens))
    check_decode(out, lse, want)


@pytest.mark.parametrize("q_lens,kv_lens,heads,page,nan", [
    ([7, 8, 9, 0, 3], [7, 64, 200, 50, 0], 16, 16, True),         # eight tokens to a tile
    ([5, 1, 2], [2, 33, 65], 48, 1, True),                        # two tokens, 32 rows empty; rows that see nothing
    ([5, 1, 2], [2, 33, 65], 64, 5, False),
    ([3, 2], [600, 31], 80, 64, True), ([2, 3], [90, 2], 130, 16, True)])
def test_prefill_tile_edges(q_lens, kv_lens, heads, page, nan):
    g = torch.Generator().manual_seed(sum(q_lens) * 100 + heads)
    cpu = paged(g, kv_lens, page, heads, sum(q_lens))
    cpu["qo_indptr"] = torch.tensor([sum(q_lens[:i]) for i in range(len(q_lens) + 1)], dtype=torch.int32)
    want = attention.causal_prefill_reference(cpu, mla=True, paged=True, page_size=page, nan_for_masked=nan, per_head_loop=False)
    out, lse = run(cpu, mla=True, paged=True, nan=nan, max_kv_len=max(kv_lens))
    check(out, lse, want)
