"""A workspace made for a call of more rows serves a call of fewer: the parts that rows of a last round are cut into
are worth having, but no call needs them."""
import ctypes

import pytest
import torch

from dsa_triton_ascend_b200 import _cabi, _host, check_status, sparse_flash_attention_triton
from dsa_triton_ascend_b200 import dense_loss_backward as dense_loss
from dsa_triton_ascend_b200 import sparse_flash_attention_grad as sfa_grad
from dsa_triton_ascend_b200 import sparse_lightning_indexer_grad_kl_loss as sparse_loss

FEW, MANY, SLOTS, HEADS = 222, 296, 2048, 64     # 74 items for a round of 148 SMs are cut in two, none are left of 296


def _bytes(name, p):
    n = ctypes.c_size_t(0)
    p.struct_size = ctypes.sizeof(p)
    for field, kind in p._fields_:
        if kind is ctypes.c_void_p and not getattr(p, field) and field not in ("seq_q", "seq_k"):
            setattr(p, field, 256)
    assert getattr(_cabi.lib, name)(ctypes.byref(p), ctypes.byref(n)) == 0
    return n.value


def _attention(rows, dtype):
    p = _cabi.DsaSfaGradParams()
    p.batch, p.s1, p.s2, p.n1, p.d, p.d_rope, p.key_rows = 1, rows, SLOTS + 48, HEADS, 512, 64, SLOTS + 48
    p.sparse_count, p.sparse_block_size, p.sparse_mode, p.dtype = SLOTS, 1, 0, dtype
    return p


@pytest.mark.parametrize("dtype", [_cabi.DTYPE_BF16, _cabi.DTYPE_FP16])
def test_attention_sizes_grow_with_the_rows(dtype):
    uncut = [_bytes("dsa_sfa_grad_workspace_bytes_uncut", _attention(r, dtype)) for r in range(1, 600)]
    whole = [_bytes("dsa_sfa_grad_workspace_bytes", _attention(r, dtype)) for r in range(1, 600)]
    assert all(a < b for a, b in zip(uncut, uncut[1:])) and all(a <= b for a, b in zip(uncut, whole))
    assert whole[FEW - 1] > whole[MANY - 1] == uncut[MANY - 1]


def _loss(rows, dtype, dense):
    p = _cabi.DsaSliGradParams()
    p.batch, p.s1, p.s2, p.n1, p.n2, p.d, p.g, p.d_idx = 1, rows, SLOTS + 48, 16, 1, 128, HEADS, 128
    p.topk, p.dense, p.dtype, p.dtype_w = SLOTS, int(dense), dtype, dtype
    return p


@pytest.mark.parametrize("dense", [False, True])
def test_loss_sizes_grow_with_the_rows(dense):
    uncut = [_bytes("dsa_sli_grad_workspace_bytes_uncut", _loss(r, 0, dense)) for r in range(1, 600)]
    whole = [_bytes("dsa_sli_grad_workspace_bytes", _loss(r, 0, dense)) for r in range(1, 600)]
    assert all(a < b for a, b in zip(uncut, uncut[1:])) and all(a <= b for a, b in zip(uncut, whole))
    assert whole[FEW - 1] > whole[MANY - 1] == uncut[MANY - 1]


class _Sized:
    """Workspaces of a given size whatever is asked for; or the first ones refused."""
    def __init__(self, nbytes=None, refuse=0):
        self.nbytes, self.refuse, self.asked = nbytes, refuse, []

    def __call__(self, nbytes, device):
        self.asked.append(int(nbytes))
        if len(self.asked) <= self.refuse:
            raise torch.cuda.OutOfMemoryError("no room")
        ws = _host.workspace(self.nbytes or nbytes, device)
        return ws.fill_(255)          # (nothing may rely on what it holds)


def _launches(call, *args, **kw):
    before = _cabi.lib.dsa_kernel_launch_count()
    out = call(*args, **kw)
    check_status()
    return out, _cabi.lib.dsa_kernel_launch_count() - before


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_attention_backward(dtype, monkeypatch):
    gen = torch.Generator(device="cuda").manual_seed(1)
    normal = lambda *s: (torch.randn(s, generator=gen, device="cuda") * 0.3).to(dtype)   # noqa: E731
    keys = SLOTS + 48
    q, qr, k, kr = normal(1, FEW, HEADS, 512), normal(1, FEW, HEADS, 64), normal(1, keys, 1, 512), normal(1, keys, 1, 64)
    idx = torch.rand(FEW, keys, generator=gen, device="cuda").argsort(1)[:, :SLOTS].to(torch.int32).view(1, FEW, 1, SLOTS)
    kw = dict(scale_value=1.0 / 24.0, query_rope=qr, key_rope=kr, sparse_mode=0)
    out, mx, sm = sparse_flash_attention_triton(q, k, k, idx, return_softmax_lse=True, **kw)

    d_out = normal(1, FEW, HEADS, 512)

    def call():
        return _launches(sfa_grad.sparse_flash_attention_grad_triton, q, k, k, idx, d_out, out, mx, sm, **kw)

    cut, cut_launches = call()
    code = _cabi.DTYPE_BF16 if dtype == torch.bfloat16 else _cabi.DTYPE_FP16
    larger = _Sized(_bytes("dsa_sfa_grad_workspace_bytes", _attention(MANY, code)))
    monkeypatch.setattr(sfa_grad, "workspace", larger)
    got, launches = call()
    # (on mma.sync there would be two kernels in all)
    assert larger.nbytes < larger.asked[0] and 2 < launches <= cut_launches
    scarce = _Sized(refuse=1)
    monkeypatch.setattr(sfa_grad, "workspace", scarce)
    again, launches = call()
    assert len(scarce.asked) == 2 and scarce.asked[1] < scarce.asked[0] and 2 < launches <= cut_launches
    for i in (0, 3):                                     # d_query, d_query_rope: whole rows, no atomics
        assert torch.equal(got[i], again[i])
    bound = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)       # one rounding of an fp32 sum on each side
    for a, b in zip(got, cut):
        assert (a.double() - b.double()).norm() <= bound * b.double().norm()


@pytest.mark.gpu
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_indexer_losses(dtype, dense, monkeypatch):
    gen = torch.Generator(device="cuda").manual_seed(2)
    normal = lambda *s: (torch.randn(s, generator=gen, device="cuda") * 0.3).to(dtype)   # noqa: E731
    keys = SLOTS + 48
    q, k, qi, ki = normal(1, FEW, 16, 128), normal(1, keys, 1, 128), normal(1, FEW, HEADS, 128), normal(1, keys, 1, 128)
    w = normal(1, FEW, HEADS).abs()
    x = torch.einsum("shd,kd->shk", q[0].float(), k[0, :, 0].float()) / 128 ** 0.5
    mx = x.amax(-1).view(1, 1, FEW, 16)
    sm = (x - x.amax(-1, keepdim=True)).exp().sum(-1).view(1, 1, FEW, 16)
    idx = torch.rand(FEW, keys, generator=gen, device="cuda").argsort(1)[:, :SLOTS].to(torch.int32).view(1, FEW, 1, SLOTS)
    module = dense_loss if dense else sparse_loss
    top, total = dense_loss.npu_dense_lightning_indexer_softmax_lse_triton(qi, ki, w)

    def call():
        if dense:
            return _launches(dense_loss.dense_loss_backward_triton, q, k, qi, ki, w, mx, sm, top, total, 128 ** -0.5)
        return _launches(sparse_loss.sparse_lightning_indexer_grad_kl_loss_triton, q, k, qi, ki, w, idx, mx, sm,
                         scale_value=128 ** -0.5)

    cut, cut_launches = call()
    code = _cabi.DTYPE_BF16 if dtype == torch.bfloat16 else _cabi.DTYPE_FP16
    larger = _Sized(_bytes("dsa_sli_grad_workspace_bytes", _loss(MANY, code, dense)))
    monkeypatch.setattr(module, "workspace", larger)
    got, launches = call()
    assert larger.nbytes < larger.asked[0] and launches <= cut_launches
    scarce = _Sized(refuse=1)
    monkeypatch.setattr(module, "workspace", scarce)
    again, launches = call()
    assert len(scarce.asked) == 2 and scarce.asked[1] < scarce.asked[0] and launches <= cut_launches
    for i in (0, 2):                                     # d_query_index, d_weights: whole rows, no atomics
        assert torch.equal(got[i], again[i])
    bound = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)       # one rounding of an fp32 sum on each side
    for a, b in zip(got, cut):
        assert (a.double() - b.double()).norm() <= bound * b.double().norm()
