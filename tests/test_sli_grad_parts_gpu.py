"""Indexer loss gradients where the last round of work items is cut into parts: rows do not depend on each other, so
the last rows of a call that is cut have to come out as in a shorter call that is not."""
import ctypes

import pytest
import torch

from dsa_triton_ascend_b200 import _cabi, _host
from dsa_triton_ascend_b200 import dense_loss_backward as dense_loss
from dsa_triton_ascend_b200 import sparse_lightning_indexer_grad_kl_loss as sparse_loss
from dsa_triton_ascend_b200 import (check_status, dense_lightning_indexer_softmax_lse_triton, dense_loss_backward_triton,
                                    sparse_lightning_indexer_grad_kl_loss_triton)

pytestmark = pytest.mark.gpu


def _parts(rows, keys, heads, slots, dense):
    """Parts that the items of a call's last round are cut into, from the size of its workspace."""
    p = _cabi.DsaSliGradParams()
    p.struct_size = ctypes.sizeof(p)
    for name, kind in p._fields_:
        if kind is ctypes.c_void_p and name not in ("seq_q", "seq_k"):
            setattr(p, name, 256)
    p.batch, p.s1, p.s2, p.n1, p.n2, p.d, p.g, p.d_idx = rows, 1, keys, 16, 1, 128, heads, 128
    p.topk, p.dense = slots, int(dense)
    total, uncut = ctypes.c_size_t(0), ctypes.c_size_t(0)
    assert _cabi.lib.dsa_sli_grad_workspace_bytes(ctypes.byref(p), ctypes.byref(total)) == 0
    assert _cabi.lib.dsa_sli_grad_workspace_bytes_uncut(ctypes.byref(p), ctypes.byref(uncut)) == 0
    left = rows * ((heads + 63) // 64) % 148
    return max(1, (total.value - uncut.value) // (64 * 129 * 4) // left)


# sequences of one row: `cut` of them leave `cut x blocks of 64 heads - 148` items for the last round, in `parts` parts;
# the last `whole` of them fill more than half a round by themselves.  `short`: of the last sequences some have 0 to 300
# keys and stay whole beside the others, some 1024 or 1100 (8 and 9 tiles: of four parts, two and three)
@pytest.mark.parametrize("cut,whole,heads,slots,parts,short", [
    (200, 100, 16, 1100, 2, False), (160, 100, 64, 2048, 4, False), (100, 50, 80, 1152, 2, False),
    (160, 80, 16, 520, 1, False), (160, 80, 16, 2048, 4, True), (200, 100, 64, 1100, 2, True)])
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_parts_add_up(cut, whole, heads, slots, parts, short, dense, dtype, monkeypatch):
    for module in (dense_loss, sparse_loss):
        # (what is not written before it is read shows as a NaN)
        monkeypatch.setattr(module, "workspace", lambda nbytes, device: _host.workspace(nbytes, device).fill_(255))
    gen = torch.Generator(device="cuda").manual_seed(cut + heads)

    def normal(*shape, scale=0.3):
        return (torch.randn(shape, generator=gen, device="cuda") * scale).to(dtype)

    s2 = slots if dense else slots + 100
    assert _parts(cut, s2, heads, slots, dense) == parts and _parts(whole, s2, heads, slots, dense) == 1
    lens = [s2] * cut
    if short:
        lens[-9:] = [0, 1, 300, 1100, 0, 128, 129, 1024, 2]
    q, k, qi, ki = normal(cut, 1, 16, 128), normal(cut, s2, 1, 128), normal(cut, 1, heads, 128), normal(cut, s2, 1, 128)
    w = normal(cut, 1, heads).abs()
    x = torch.einsum("bhd,bkd->bhk", q[:, 0].float(), k[:, :, 0].float()) * 128 ** -0.5
    mx = x.amax(-1).view(cut, 1, 1, 16)
    sm = (x - x.amax(-1, keepdim=True)).exp().sum(-1).view(cut, 1, 1, 16)
    idx = torch.stack([torch.randperm(s2, generator=gen, device="cuda")[:slots] for _ in range(cut)])
    idx = idx.to(torch.int32).view(cut, 1, 1, slots)

    # (taken once: the scores of more than 64 heads are added with atomics)
    top, total = dense_lightning_indexer_softmax_lse_triton(qi, ki, w, actual_seq_klen=lens)

    def call(n):
        a, b, c, d, e, m, s, i = (t[cut - n:].contiguous() for t in (q, k, qi, ki, w, mx, sm, idx))
        if not dense:
            return sparse_lightning_indexer_grad_kl_loss_triton(a, b, c, d, e, i, m, s, scale_value=128 ** -0.5,
                                                                actual_seq_klen=lens[cut - n:])[:3]
        return dense_loss_backward_triton(a, b, c, d, e, m, s, top[cut - n:], total[cut - n:], 128 ** -0.5,
                                          actual_seq_klen=lens[cut - n:])[:3]

    got, again, want = call(cut), call(cut), call(whole)
    check_status()
    bound = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)      # one rounding of an fp32 sum on each side
    for g, r in zip(got, want):
        g, r = g[cut - whole:].double(), r.double()
        assert r.norm() > 0 and (g - r).norm() <= bound * r.norm()
    assert torch.equal(got[0], again[0]) and torch.equal(got[2], again[2])     # no atomics in dQI and dW


@pytest.mark.parametrize("rows,keys,cut", [(222, 640, False), (222, 768, True), (20, 640, False), (20, 768, True)])
@pytest.mark.parametrize("dense", [False, True])
def test_short_rows_stay_whole(rows, keys, cut, dense, monkeypatch):
    """Parts are made of the keys that a row has, whatever the width of its list: 5 or 6 tiles of 128 keys here, of 2048
    slots or more.  The workspace shows whether any part left a sum."""
    gen = torch.Generator(device="cuda").manual_seed(rows)
    normal = lambda *s: (torch.randn(s, generator=gen, device="cuda") * 0.3).bfloat16()   # noqa: E731
    s2 = 2048 if dense else 2100
    q, k, qi, ki = normal(1, rows, 16, 128), normal(1, s2, 1, 128), normal(1, rows, 64, 128), normal(1, s2, 1, 128)
    w = normal(1, rows, 64).abs()
    mx, sm = torch.zeros(1, 1, rows, 16, device="cuda"), torch.full((1, 1, rows, 16), float(keys), device="cuda")
    idx = torch.arange(2048, dtype=torch.int32, device="cuda").repeat(1, rows, 1, 1).view(1, rows, 1, 2048)
    lens = [keys]

    top, total = dense_lightning_indexer_softmax_lse_triton(qi, ki, w, actual_seq_klen=lens)
    held = []

    def marked(nbytes, device):
        held.append(_host.workspace(nbytes, device).fill_(255))
        return held[-1]

    for module in (dense_loss, sparse_loss):
        monkeypatch.setattr(module, "workspace", marked)

    def call():
        if dense:
            return dense_loss_backward_triton(q, k, qi, ki, w, mx, sm, top, total, 128 ** -0.5, actual_seq_klen=lens)
        return sparse_lightning_indexer_grad_kl_loss_triton(q, k, qi, ki, w, idx, mx, sm, scale_value=128 ** -0.5,
                                                            actual_seq_klen=lens)

    got = call()
    check_status()
    left = rows % 148
    size = left * min(4, 148 // left) * 64 * 129 * 4        # of the parts, at the end of the workspace
    assert bool((held[0][-size:] != 255).any()) == cut
    for module in (dense_loss, sparse_loss):
        monkeypatch.setattr(module, "workspace", lambda nbytes, device: _host.workspace(nbytes - size, device).fill_(255))
    want = call()                                           # whole rows
    bound = 2.0 ** -8                                       # one rounding to bf16 on each side
    for i in range(3):
        assert (got[i].double() - want[i].double()).norm() <= bound * want[i].double().norm()
        if not cut and i != 1:                              # (d_key_index: atomics)
            assert torch.equal(got[i], want[i])
