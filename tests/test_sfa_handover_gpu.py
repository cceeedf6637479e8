"""Attention forward over CTA pairs: keys and values that one CTA's warps copied are read by products that the other
CTA issues.  A hand-over that let a product start early would change single tiles from run to run."""
import pytest
import torch

from dsa_triton_ascend_b200 import check_status, sparse_flash_attention_triton
from dsa_triton_ascend_b200 import sparse_flash_attention as sfa

pytestmark = pytest.mark.gpu


# many tiles per token on every pair; one tile per token; split along the keys; a last tile of one key
@pytest.mark.parametrize("rows,keys,count", [(592, 4096, 2048), (1184, 96, 64), (3, 4096, 2048), (300, 700, 577)])
@pytest.mark.parametrize("heads", [16, 65, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_repeats_bit_for_bit(rows, keys, count, heads, dtype):
    gen = torch.Generator(device="cuda").manual_seed(rows + heads)

    def normal(*shape):
        return torch.randn(shape, generator=gen, device="cuda").to(dtype)

    q, qr, k, kr = normal(1, rows, heads, 512), normal(1, rows, heads, 64), normal(1, keys, 1, 512), normal(1, keys, 1, 64)
    idx = torch.rand(rows, keys, generator=gen, device="cuda").argsort(1)[:, :count].to(torch.int32).view(1, rows, 1, count)
    kw = dict(scale_value=576 ** -0.5, query_rope=qr, key_rope=kr, sparse_mode=0, return_softmax_lse=True)
    first = sparse_flash_attention_triton(q, k, k, idx, **kw)
    for _ in range(20):
        for a, b in zip(first, sparse_flash_attention_triton(q, k, k, idx, **kw)):
            assert torch.equal(a, b)
    check_status()
    sfa.set_kernel("portable")
    try:
        want = sparse_flash_attention_triton(q, k, k, idx, **kw)
    finally:
        sfa.set_kernel("auto")
    # P and the output are rounded to the io dtype on both sides (half an ulp each): two ulp of the largest value
    ulp = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert (first[0].double() - want[0].double()).abs().max() <= 2 * ulp * want[0].double().abs().max()
