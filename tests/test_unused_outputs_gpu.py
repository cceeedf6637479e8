"""Outputs that were not asked for are zeros, whatever the memory held before: the kernels store them."""
import pytest
import torch

from dsa_triton_ascend_b200 import check_status, lightning_indexer_triton, sparse_flash_attention_triton
from dsa_triton_ascend_b200 import lightning_indexer as li, sparse_flash_attention as sfa

pytestmark = pytest.mark.gpu


def _dirty(nbytes):
    """Leave blocks of ones of this size in the allocator's cache for the call's outputs to land in."""
    blocks = [torch.full((max(nbytes, 1),), 255, dtype=torch.uint8, device="cuda") for _ in range(4)]
    del blocks


# rows of up to 8192 keys and longer ones, io-dtype and fp32 ranking, 16-byte and odd output rows, keys outnumbered
@pytest.mark.parametrize("keys,k,rank", [(300, 64, "io_dtype"), (300, 7, "io_dtype"), (40, 65, "io_dtype"),
                                         (9000, 128, "io_dtype"), (300, 64, "fp32"), (300, 2050, "io_dtype")])
@pytest.mark.parametrize("kernel", ["auto", "portable"])
def test_indexer_values(keys, k, rank, kernel):
    q = torch.randn(1, 5, 8, 128, device="cuda").bfloat16()
    key = torch.randn(1, keys, 1, 128, device="cuda").bfloat16()
    w = torch.randn(1, 5, 8, device="cuda")
    li.set_kernel(kernel)
    li.set_rank_mode(rank)
    try:
        _dirty(5 * k * 2)
        _, values = lightning_indexer_triton(q, key, w, sparse_count=k)
        check_status()
    finally:
        li.set_kernel("auto")
        li.set_rank_mode("io_dtype")
    assert values.shape == (1, 5, 1, k) and not values.view(torch.int16).any()


@pytest.mark.parametrize("rows,heads,kernel", [(3, 128, "auto"), (3, 16, "auto"), (600, 17, "auto"), (3, 5, "auto"),
                                               (3, 16, "portable")])
@pytest.mark.parametrize("count", [6, 64])
def test_attention_statistics(rows, heads, kernel, count):
    q, qr = (torch.randn(1, rows, heads, d, device="cuda").bfloat16() for d in (512, 64))
    k, kr = (torch.randn(1, rows + 64, 1, d, device="cuda").bfloat16() for d in (512, 64))
    idx = torch.arange(count, dtype=torch.int32, device="cuda").expand(1, rows, 1, count)
    sfa.set_kernel(kernel)
    try:
        _dirty(rows * heads * 4)
        _, mx, sm = sparse_flash_attention_triton(q, k, k, idx, query_rope=qr, key_rope=kr, sparse_mode=3)
        check_status()
    finally:
        sfa.set_kernel("auto")
    for t in (mx, sm):
        assert t.shape == (1, 1, rows, heads) and not t.view(torch.int32).any()
