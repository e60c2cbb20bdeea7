"""Block-scaled GEMM on either side of each line of its dispatch: the weight-streaming kernel (up to 16 rows, each way of
splitting K over a CTA's warps), tiles of 128 columns whose K two or four CTAs share, tiles of 256 columns, an item
to a CTA, several in turn, and drawn from the work-item counter.  Oracle and tolerance of test_gpu_gemm.py."""
import pytest
import torch

from oracle import compare
from test_gpu_gemm import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [
    (1, 128, 128), (8, 8192, 256), (9, 4096, 640), (16, 1024, 1152),                 # weight streaming
    (17, 128, 1024), (64, 384, 2048), (129, 640, 2176), (300, 1536, 1152),           # shared K
    (17, 384, 896), (130, 9600, 1024), (1025, 4096, 256),                            # whole K, an item to a CTA at most
    (2500, 4096, 128), (2500, 4224, 640), (1100, 9600, 1024), (6000, 5120, 128)])    # several items to a CTA in turn, odd and even K blocks; counter
def test_dispatch_edges(m, n, k):
    if m in (2500, 1100, 6000):          # what those are for: in turn up to six items a CTA, from the counter beyond
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        items = -(-m // 128) * -(-n // 256)
        assert sms < items <= 6 * sms if m < 6000 else items > 6 * sms
    c, want = run(m, n, k)
    ok, bad, err = compare.compare(c, want, atol=2e-2, rtol=2e-2)
    assert ok, f"{bad} mismatches, max abs err {err}"
    assert compare.rel_frobenius(c, want) <= 1e-2
