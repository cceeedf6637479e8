"""Attention backward where the last round of work items is cut into parts: against the CUDA-core kernel, which takes
every row as a whole."""
import ctypes

import pytest
import torch

from dsa_triton_ascend_b200 import _cabi, _host, check_status, sparse_flash_attention_grad_triton, sparse_flash_attention_triton
from dsa_triton_ascend_b200 import sparse_flash_attention_grad as grad

pytestmark = pytest.mark.gpu


def _parts(rows, keys, heads, count, left, dtype):
    """Parts that the call's `left` last items are cut into, from the size of its workspace."""
    p = _cabi.DsaSfaGradParams()
    p.struct_size = ctypes.sizeof(p)
    for name, kind in p._fields_:
        if kind is ctypes.c_void_p and name not in ("seq_q", "seq_k"):
            setattr(p, name, 256)
    p.batch, p.s1, p.s2, p.n1, p.d, p.d_rope, p.key_rows = 1, rows, keys, heads, 512, 64, keys
    p.sparse_count, p.sparse_block_size, p.sparse_mode = count, 1, 3
    p.dtype = _cabi.DTYPE_BF16 if dtype == torch.bfloat16 else _cabi.DTYPE_FP16
    total, uncut = ctypes.c_size_t(0), ctypes.c_size_t(0)
    assert _cabi.lib.dsa_sfa_grad_workspace_bytes(ctypes.byref(p), ctypes.byref(total)) == 0
    assert _cabi.lib.dsa_sfa_grad_workspace_bytes_uncut(ctypes.byref(p), ctypes.byref(uncut)) == 0
    return max(1, (total.value - uncut.value) // (64 * 576 * 4) // left)


# items of 64 heads left for the last round of 148 and the parts they are cut into: 2 in four; 52 in two; 2 of two head
# blocks (the second of 16 heads), in three; 49 in three, of which 20 have 61 to 80 keys (2 tiles: two parts and
# none in the place of the third) and the last 20 have 0 to 12 (whole); 75, more than half a round, as they are
@pytest.mark.parametrize("q_lens,k_lens,heads,count,left,parts", [
    ([150], [1700], 16, 1536, 2, 4), ([200], [1200], 64, 1152, 52, 2), ([75], [1300], 80, 1152, 2, 3),
    ([157, 20, 20], [1000, 80, 12], 16, 1152, 49, 3), ([223], [1200], 16, 1152, 75, 1)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_parts_add_up(q_lens, k_lens, heads, count, left, parts, dtype, monkeypatch):
    assert _parts(sum(q_lens), sum(k_lens), heads, count, left, dtype) == parts
    # (what is not written before it is read shows as a NaN)
    monkeypatch.setattr(grad, "workspace", lambda nbytes, device: _host.workspace(nbytes, device).fill_(255))
    gen = torch.Generator(device="cuda").manual_seed(sum(q_lens) + heads)
    rows, keys = sum(q_lens), sum(k_lens)

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


@pytest.mark.parametrize("rows,keys,cut", [(222, 144, False), (222, 192, True), (20, 48, False), (20, 96, True)])
def test_short_rows_stay_whole(rows, keys, cut, monkeypatch):
    """Parts are made of the keys that a row has, whatever the width of its list: 1 to 4 tiles of 48 keys here, of 2048
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
