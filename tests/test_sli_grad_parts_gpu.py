"""Indexer loss gradients where the last round of work items is cut into parts: rows do not depend on each other, so
the last rows of a call that is cut have to come out as in a shorter call that is not."""
import pytest
import torch

from dsa_triton_ascend_b200 import _host
from dsa_triton_ascend_b200 import dense_loss_backward as dense_loss
from dsa_triton_ascend_b200 import sparse_lightning_indexer_grad_kl_loss as sparse_loss
from dsa_triton_ascend_b200 import (check_status, dense_lightning_indexer_softmax_lse_triton, dense_loss_backward_triton,
                                    sparse_lightning_indexer_grad_kl_loss_triton)

pytestmark = pytest.mark.gpu


# sequences of one row: `cut` of them leave `cut x blocks of 64 heads - 148` items for the last round (52: two parts, 12:
# four), the last `whole` of them fill more than half a round by themselves.  520 slots: parts without keys
@pytest.mark.parametrize("cut,whole,heads,slots", [(200, 100, 16, 1100), (160, 100, 64, 2048), (100, 50, 80, 1152),
                                                   (160, 80, 16, 520)])
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_parts_add_up(cut, whole, heads, slots, dense, dtype):
    gen = torch.Generator(device="cuda").manual_seed(cut + heads)

    def normal(*shape, scale=0.3):
        return (torch.randn(shape, generator=gen, device="cuda") * scale).to(dtype)

    s2 = slots if dense else slots + 100
    q, k, qi, ki = normal(cut, 1, 16, 128), normal(cut, s2, 1, 128), normal(cut, 1, heads, 128), normal(cut, s2, 1, 128)
    w = normal(cut, 1, heads).abs()
    x = torch.einsum("bhd,bkd->bhk", q[:, 0].float(), k[:, :, 0].float()) * 128 ** -0.5
    mx = x.amax(-1).view(cut, 1, 1, 16)
    sm = (x - x.amax(-1, keepdim=True)).exp().sum(-1).view(cut, 1, 1, 16)
    idx = torch.stack([torch.randperm(s2, generator=gen, device="cuda")[:slots] for _ in range(cut)])
    idx = idx.to(torch.int32).view(cut, 1, 1, slots)

    top, total = dense_lightning_indexer_softmax_lse_triton(qi, ki, w)    # (more than 64 heads are added with atomics)

    def call(n):
        a, b, c, d, e, m, s, i = (t[cut - n:].contiguous() for t in (q, k, qi, ki, w, mx, sm, idx))
        if not dense:
            return sparse_lightning_indexer_grad_kl_loss_triton(a, b, c, d, e, i, m, s, scale_value=128 ** -0.5)[:3]
        return dense_loss_backward_triton(a, b, c, d, e, m, s, top[cut - n:], total[cut - n:], 128 ** -0.5)[:3]

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
