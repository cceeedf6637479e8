"""Attention backward where the last round of work items is cut into parts: against the CUDA-core kernel, which takes
every row as a whole."""
import pytest
import torch

from dsa_triton_ascend_b200 import _host, check_status, sparse_flash_attention_grad_triton, sparse_flash_attention_triton
from dsa_triton_ascend_b200 import sparse_flash_attention_grad as grad

pytestmark = pytest.mark.gpu


# items of 64 heads left for the last round of 148: 2 (four parts), 52 (two parts), 2 of two head blocks
# (the second of 16 heads), 49 (three parts, short rows: parts without keys), 75 (whole: more than half a round)
@pytest.mark.parametrize("q_lens,k_lens,heads", [([150], [1200], 16), ([200], [1200], 64), ([75], [1300], 80),
                                                 ([20, 177], [20, 1000], 16), ([223], [1200], 16)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_parts_add_up(q_lens, k_lens, heads, dtype):
    gen = torch.Generator(device="cuda").manual_seed(sum(q_lens) + heads)
    rows, keys, count = sum(q_lens), sum(k_lens), 1152

    def normal(*shape):
        return (torch.randn(shape, generator=gen, device="cuda") * 0.3).to(dtype)

    q, qr, k, kr = normal(rows, heads, 512), normal(rows, heads, 64), normal(keys, 1, 512), normal(keys, 1, 64)
    d_out = normal(rows, heads, 512)
    ends_q, ends_k = ([sum(v[:i + 1]) for i in range(len(v))] for v in (q_lens, k_lens))
    idx = torch.stack([torch.randperm(max(k_lens), generator=gen, device="cuda")[:count] if max(k_lens) >= count else
                       torch.nn.functional.pad(torch.randperm(max(k_lens), generator=gen, device="cuda"),
                                               (0, count - max(k_lens)), value=-1) for _ in range(rows)])
    idx = idx.to(torch.int32).view(rows, 1, count)
    kw = dict(scale_value=576 ** -0.5, query_rope=qr, key_rope=kr, actual_seq_lengths_query=ends_q,
              actual_seq_lengths_kv=ends_k, sparse_mode=3)
    out, mx, sm = sparse_flash_attention_triton(q, k, k, idx, layout_query="TND", layout_kv="TND",
                                                return_softmax_lse=True, **kw)
    args = (q, k, k, idx, d_out, out, mx, sm)
    got = sparse_flash_attention_grad_triton(*args, layout="TND", **kw)
    again = sparse_flash_attention_grad_triton(*args, layout="TND", **kw)
    check_status()
    grad.set_kernel("portable")
    try:
        want = sparse_flash_attention_grad_triton(*args, layout="TND", **kw)
    finally:
        grad.set_kernel("auto")
    # each side rounds an fp32 sum once: 2^-9 (bf16) or 2^-12 (fp16) of a value at most
    bound = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    for g, w in zip(got, want):
        assert (g.double() - w.double()).norm() <= bound * w.double().norm()
    assert torch.equal(got[0], again[0]) and torch.equal(got[3], again[3])     # d_query, d_query_rope: no atomics


@pytest.mark.parametrize("rows,keys,cut", [(222, 240, False), (222, 288, True), (20, 48, False), (20, 96, True)])
def test_short_rows_stay_whole(rows, keys, cut, monkeypatch):
    """Parts are made of the keys that a row has, whatever the width of its list: 1 to 6 tiles of 48 keys here, of 2048
    slots.  The workspace shows whether any part left a sum."""
    held = []

    def marked(nbytes, device):
        held.append(_host.workspace(nbytes, device).fill_(255))
        return held[-1]

    monkeypatch.setattr(grad, "workspace", marked)
    gen = torch.Generator(device="cuda").manual_seed(rows)
    normal = lambda *s: (torch.randn(s, generator=gen, device="cuda") * 0.3).bfloat16()   # noqa: E731
    q, qr, k, kr, d_out = (normal(1, n, h, d) for n, h, d in ((rows, 64, 512), (rows, 64, 64), (keys, 1, 512), (keys, 1, 64),
                                                               (rows, 64, 512)))
    idx = torch.full((1, rows, 1, 2048), -1, dtype=torch.int32, device="cuda")
    idx[..., :keys] = torch.arange(keys, device="cuda")
    kw = dict(scale_value=576 ** -0.5, query_rope=qr, key_rope=kr, sparse_mode=0)
    out, mx, sm = sparse_flash_attention_triton(q, k, k, idx, return_softmax_lse=True, **kw)
    got = sparse_flash_attention_grad_triton(q, k, k, idx, d_out, out, mx, sm, **kw)
    check_status()
    left = rows % 148
    size = left * min(4, 148 // left) * 64 * 576 * 4        # of the parts, at the end of the workspace
    assert bool((held[0][-size:] != 255).any()) == cut
    grad.set_kernel("portable")
    try:
        want = sparse_flash_attention_grad_triton(q, k, k, idx, d_out, out, mx, sm, **kw)
    finally:
        grad.set_kernel("auto")
    for g, w in zip(got, want):
        assert (g.double() - w.double()).norm() <= 2.0 ** -8 * w.double().norm()    # one rounding to bf16 each
