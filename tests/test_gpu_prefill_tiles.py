"""Causal GQA prefill at the sizes where its tiles can go wrong: query lengths and KV lengths on either side of a tile's
edge, every number of query heads per KV head, segments without query or KV rows, rows that see nothing, and the form
that runs a decode sequence per query row (a few rows behind a long prefix).  Oracle and tolerance of test_gpu_prefill.py."""
import pytest
import torch

from oracle import attention
from test_gpu_prefill import check, run

pytestmark = pytest.mark.gpu


def problem(seed, q_lens, kv_lens, heads, kv_heads, page):
    """Paged with pages of ``page`` rows, or ragged when ``page`` is 0."""
    g = torch.Generator().manual_seed(seed)
    q_lens, kv_lens = torch.tensor(q_lens), torch.tensor(kv_lens)
    zero = torch.zeros(1, dtype=torch.long)
    cpu = {"q": torch.randn((int(q_lens.sum()), heads, 128), generator=g).to(torch.bfloat16),
           "qo_indptr": torch.cat([zero, q_lens.cumsum(0)]).int(), "sm_scale": torch.tensor([128.0 ** -0.5])}
    if page:
        pages = (kv_lens + page - 1) // page
        pool = int(pages.sum()) + 3
        cpu["kv_indptr"] = torch.cat([zero, pages.cumsum(0)]).int()
        cpu["kv_indices"] = torch.randperm(pool, generator=g)[:int(pages.sum())].int()
        cpu["kv_last_page_len"] = torch.where(pages > 0, kv_lens - (pages - 1) * page, torch.zeros_like(kv_lens)).int()
        shape, names = (pool, page, kv_heads, 128), ("k_cache", "v_cache")
    else:
        cpu["kv_indptr"] = torch.cat([zero, kv_lens.cumsum(0)]).int()
        shape, names = (int(kv_lens.sum()), kv_heads, 128), ("k", "v")
    for name in names:
        cpu[name] = torch.randn(shape, generator=g).to(torch.bfloat16)
    return cpu


@pytest.mark.parametrize("q_lens,kv_lens,heads,kv_heads,page,nan", [
    ([63, 64, 65], [127, 128, 129], 8, 2, 16, True),              # G = 4: 32 tokens to a row tile, 64 to a CTA
    ([1, 31, 33, 0, 7], [1, 300, 40, 50, 0], 8, 2, 5, False),     # half-empty tiles; no query rows; no KV rows
    ([130, 300], [100, 300], 4, 4, 0, True),                      # G = 1: rows that see nothing (30 of the first segment)
    ([130, 20], [100, 257], 4, 4, 64, False),                     # the same as zeros
    ([33, 17, 85], [256, 255, 90], 3, 1, 1, True),                # G = 3: 42 tokens, two rows of a tile stay empty
    ([26, 51], [26, 385], 5, 1, 16, True), ([21, 43], [400, 43], 6, 1, 0, True), ([19, 37], [129, 700], 14, 2, 16, False),
    ([16, 33], [513, 64], 16, 2, 16, True),                       # G = 8
    ([2, 1], [6000, 4097], 8, 1, 16, True),                       # one decode sequence per query row
    # tiles that are cut into pieces of KV tiles: rows that see every piece and the first ones only, few rows, rows that see nothing
    ([64], [3000], 8, 2, 16, False), ([40, 3, 0], [2500, 900, 0], 16, 2, 5, True), ([5], [1300], 64, 8, 64, False),
    ([130, 20, 200], [100, 2000, 300], 4, 4, 0, True), ([300, 7, 64], [290, 1025, 1024], 8, 1, 0, True), ([70], [4000], 3, 3, 16, True),
    ([900], [800], 4, 2, 0, True),                                # pieces of which some rows see nothing
])
def test_tile_edges(q_lens, kv_lens, heads, kv_heads, page, nan):
    cpu = problem(len(q_lens) * 100 + heads, q_lens, kv_lens, heads, kv_heads, page)
    want = attention.causal_prefill_reference(cpu, mla=False, paged=page > 0, page_size=page or 1, nan_for_masked=nan, per_head_loop=False)
    out, lse = run(cpu, mla=False, paged=page > 0, nan=nan, max_kv_len=max(kv_lens))
    check(out, lse, want)
