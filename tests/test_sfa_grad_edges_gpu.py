"""Attention backward where its inputs leave the ordinary: selected keys that do not exist, keys and heads whose
values are far from the others', rows without statistics.  Each call is compared with one that has to give the
same result, or with the numpy oracle."""
import ctypes
import math

import numpy as np
import pytest
import torch

from oracle import sparse_flash_attention_grad_oracle, sparse_flash_attention_oracle
from oracle.compare import sfa_grad_acceptance_rule
from oracle.inputs import sfa_grad_inputs, sparse_indices
from tests.util import dev, host, tdtype

pytestmark = pytest.mark.gpu
NAMES = ("d_query", "d_key", "d_value", "d_query_rope", "d_key_rope")


def _randn(seed, *shape, dtype, scale=0.3):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


@pytest.mark.parametrize("dtype", ["bf16", "fp16"])
@pytest.mark.parametrize("N1,K", [(64, 160), (16, 160), (64, 161)])   # 161: rows off their 16-byte boundaries
def test_selected_keys_past_the_key_tensor_take_no_part(N1, K, dtype):
    """TND key lengths that overrun the tensor: a slot that names a row which does not exist is as good as an
    unused one (-1), in whole tiles of keys too."""
    from dsa_triton_ascend_b200 import sparse_flash_attention_grad_triton
    dt = tdtype(dtype)
    T1, T2, ends_q, ends_k = 6, 100, [2, 6], [60, 200]       # keys 40.. of the second sequence do not exist
    q, qr = _randn(1, T1, N1, 512, dtype=dt), _randn(2, T1, N1, 64, dtype=dt)
    k, kr = _randn(3, T2, 1, 512, dtype=dt), _randn(4, T2, 1, 64, dtype=dt)
    do, out = _randn(5, T1, N1, 512, dtype=dt), _randn(6, T1, N1, 512, dtype=dt)
    mx, sm = torch.zeros(1, T1, N1, device="cuda"), torch.full((1, T1, N1), 150.0, device="cuda")
    rng = np.random.RandomState(7)
    idx = np.full((T1, 1, K), -1, np.int32)
    for t in range(T1):
        n = 60 if t < 2 else 140
        idx[t, 0, :n] = rng.permutation(n)
    exists = idx.copy()
    exists[2:][exists[2:] >= 40] = -1
    kw = dict(scale_value=1.0 / 24.0, query_rope=qr, key_rope=kr, actual_seq_lengths_query=ends_q,
              actual_seq_lengths_kv=ends_k, layout="TND", sparse_mode=0)
    got = sparse_flash_attention_grad_triton(q, k, k, torch.from_numpy(idx).cuda(), do, out, mx, sm, **kw)
    ref = sparse_flash_attention_grad_triton(q, k, k, torch.from_numpy(exists).cuda(), do, out, mx, sm, **kw)
    for n, a, b in zip(NAMES, got, ref):
        if n.startswith("d_query"):
            assert torch.equal(a, b), n
        else:                       # (reductions arrive in any order: one rounding of the output apart)
            sfa_grad_acceptance_rule(host(a), host(b), dtype, name=n, ulps=1.0)


def _fp16_case(seed, S1, S2, N1, K, valid, do_scale):
    """BSND inputs of which keys 0..valid-1 are in use, and forward statistics that fit them."""
    from dsa_triton_ascend_b200 import sparse_flash_attention_triton
    dt = torch.float16
    q, qr = _randn(seed, 1, S1, N1, 512, dtype=dt), _randn(seed + 1, 1, S1, N1, 64, dtype=dt)
    k, kr = _randn(seed + 2, 1, S2, 1, 512, dtype=dt), _randn(seed + 3, 1, S2, 1, 64, dtype=dt)
    do = _randn(seed + 4, 1, S1, N1, 512, dtype=dt, scale=do_scale)
    rng = np.random.RandomState(seed)
    idx = torch.from_numpy(np.stack([rng.permutation(valid)[:K] for _ in range(S1)]).astype(np.int32)).cuda()
    kw = dict(scale_value=1.0 / 24.0, query_rope=qr, key_rope=kr, actual_seq_lengths_kv=[valid], sparse_mode=0)
    idx = idx.view(1, S1, 1, K)
    out, mx, sm = sparse_flash_attention_triton(q, k, k, idx, return_softmax_lse=True, **kw)
    return q, k, idx, do, out, mx, sm, kw


@pytest.mark.parametrize("do_scale", [0.3, 1e-3])
@pytest.mark.parametrize("what", [1e3, 65504.0, math.inf, math.nan])
def test_fp16_gradients_do_not_depend_on_keys_that_nobody_selected(what, do_scale):
    """Large, infinite or undefined values in padding rows and in one visible, unselected key change nothing: d_query
    stays the same bit for bit, the scattered gradients up to the order of their sums."""
    from dsa_triton_ascend_b200 import sparse_flash_attention_grad_triton
    q, k, idx, do, out, mx, sm, kw = _fp16_case(21, 5, 300, 64, 100, 260, do_scale)
    idx[idx == 11] = -1
    ref = sparse_flash_attention_grad_triton(q, k, k, idx, do, out, mx, sm, **kw)
    foreign = k.clone()
    foreign[:, 260:] = what
    foreign[:, 11] = what
    got = sparse_flash_attention_grad_triton(q, foreign, foreign, idx, do, out, mx, sm, **kw)
    for n, a, b in zip(NAMES, got, ref):
        if n.startswith("d_query"):
            assert torch.equal(a, b), n
        else:
            sfa_grad_acceptance_rule(host(a), host(b), "fp16", name=n, ulps=1.0)


@pytest.mark.parametrize("where", ["d_out", "out"])
@pytest.mark.parametrize("what", [math.inf, math.nan])
def test_fp16_heads_do_not_lose_their_scale_to_a_head_without_finite_values(what, where):
    """An Inf or NaN in d_out or out of one head: d_query of every other head is the same, bit for bit, as without
    that head (its d_out zero)."""
    from dsa_triton_ascend_b200 import sparse_flash_attention_grad_triton
    q, k, idx, do, out, mx, sm, kw = _fp16_case(31, 5, 260, 80, 100, 260, 1e-3)
    bad = 3
    do[:, :, bad] = 0
    ref = sparse_flash_attention_grad_triton(q, k, k, idx, do, out, mx, sm, **kw)
    do, out = do.clone(), out.clone()
    if where == "d_out":
        do[:, :, bad, 7] = what
    else:
        do[:, :, bad, 7] = 1e-3
        out[:, :, bad, 7] = what
    got = sparse_flash_attention_grad_triton(q, k, k, idx, do, out, mx, sm, **kw)
    others = [h for h in range(80) if h != bad]
    assert torch.equal(got[0][:, :, others], ref[0][:, :, others])
    assert torch.equal(got[3][:, :, others], ref[3][:, :, others])


def test_fp16_head_blocks_scale_apart():
    """d_out of one head four orders larger: heads of other 64-head blocks keep their d_query bit for bit."""
    from dsa_triton_ascend_b200 import sparse_flash_attention_grad_triton
    q, k, idx, do, out, mx, sm, kw = _fp16_case(41, 5, 260, 80, 100, 260, 1e-3)
    ref = sparse_flash_attention_grad_triton(q, k, k, idx, do, out, mx, sm, **kw)
    loud = do.clone()
    loud[:, :, 70] *= 1e4
    got = sparse_flash_attention_grad_triton(q, k, k, idx, loud, out, mx, sm, **kw)
    assert torch.equal(got[0][:, :, :64], ref[0][:, :, :64]) and torch.equal(got[3][:, :, :64], ref[3][:, :, :64])


def test_a_head_without_a_sum_has_no_probabilities():
    """softmax_sum = 0 and scores that overflow to +Inf: the head contributes nothing, as if its query were zero."""
    from dsa_triton_ascend_b200 import sparse_flash_attention_grad_triton
    bf, S1, S2, N1, K, dead = torch.bfloat16, 3, 120, 20, 100, 5
    q, qr = _randn(51, 1, S1, N1, 512, dtype=bf), _randn(52, 1, S1, N1, 64, dtype=bf)
    k, kr = _randn(53, 1, S2, 1, 512, dtype=bf), _randn(54, 1, S2, 1, 64, dtype=bf)
    do, out = _randn(55, 1, S1, N1, 512, dtype=bf), _randn(56, 1, S1, N1, 512, dtype=bf)
    # feature 0: 1e20 in the dead head's query and in key 3 (score 1e40); no other head uses it
    q[..., 0], do[..., 0], k[..., 0] = 0, 0, 0
    k[:, 3, 0, 0] = 1e20
    q[:, :, dead, 0] = 1e20
    mx, sm = torch.zeros(1, 1, S1, N1, device="cuda"), torch.full((1, 1, S1, N1), 100.0, device="cuda")
    sm[..., dead] = 0
    idx = torch.arange(K, dtype=torch.int32, device="cuda").expand(1, S1, 1, K).contiguous()
    kw = dict(scale_value=1.0 / 24.0, query_rope=qr, key_rope=kr, sparse_mode=0)
    got = sparse_flash_attention_grad_triton(q, k, k, idx, do, out, mx, sm, **kw)
    still = q.clone()
    still[:, :, dead] = 0
    ref = sparse_flash_attention_grad_triton(still, k, k, idx, do, out, mx, sm, **kw)
    for n, a, b in zip(NAMES, got, ref):
        if n.startswith("d_query"):
            assert torch.equal(a, b) and (a[:, :, dead] == 0).all(), n
        else:
            sfa_grad_acceptance_rule(host(a), host(b), "bf16", name=n, ulps=1.0)


@pytest.mark.parametrize("dtype", ["bf16", "fp16"])
def test_heads_past_the_last_one_add_nothing_to_d_value(dtype):
    """17 heads in a block of 64, and a key of -Inf score (probability 0 in every head): d_value stays finite and
    is what it is without that key."""
    from dsa_triton_ascend_b200 import sparse_flash_attention_grad_triton
    dt, S1, S2, N1, K = tdtype(dtype), 3, 120, 17, 100
    q, qr = _randn(61, 1, S1, N1, 512, dtype=dt), _randn(62, 1, S1, N1, 64, dtype=dt)
    k, kr = _randn(63, 1, S2, 1, 512, dtype=dt), _randn(64, 1, S2, 1, 64, dtype=dt)
    do, out = _randn(65, 1, S1, N1, 512, dtype=dt), _randn(66, 1, S1, N1, 512, dtype=dt)
    q[..., 0], k[..., 0] = -1, 0
    mx, sm = torch.zeros(1, 1, S1, N1, device="cuda"), torch.full((1, 1, S1, N1), 100.0, device="cuda")
    idx = torch.arange(K, dtype=torch.int32, device="cuda").expand(1, S1, 1, K).clone()
    kw = dict(scale_value=1.0 / 24.0, query_rope=qr, key_rope=kr, sparse_mode=0)
    far = k.clone()
    far[:, 3, 0, 0] = math.inf
    got = sparse_flash_attention_grad_triton(q, far, far, idx, do, out, mx, sm, **kw)[2]
    idx[..., 3] = -1
    ref = sparse_flash_attention_grad_triton(q, k, k, idx, do, out, mx, sm, **kw)[2]
    sfa_grad_acceptance_rule(host(got), host(ref), dtype, name="d_value", ulps=1.0)


@pytest.mark.parametrize("dtype", ["bf16", "fp16"])
def test_the_documented_least_workspace_is_enough(dtype, monkeypatch):
    """Header and accumulators alone (what the wrapper falls back to when the larger workspace cannot be had): the
    mma.sync kernel runs, with the same results up to the rounding of the outputs."""
    from dsa_triton_ascend_b200 import _host
    from dsa_triton_ascend_b200 import sparse_flash_attention_grad as module
    dt, S1, S2, N1, K = tdtype(dtype), 5, 120, 64, 100
    q, qr = _randn(71, 1, S1, N1, 512, dtype=dt), _randn(72, 1, S1, N1, 64, dtype=dt)
    k, kr = _randn(73, 1, S2, 1, 512, dtype=dt), _randn(74, 1, S2, 1, 64, dtype=dt)
    do, out = _randn(75, 1, S1, N1, 512, dtype=dt), _randn(76, 1, S1, N1, 512, dtype=dt)
    mx, sm = torch.zeros(1, 1, S1, N1, device="cuda"), torch.full((1, 1, S1, N1), 100.0, device="cuda")
    idx = torch.arange(K, dtype=torch.int32, device="cuda").expand(1, S1, 1, K).contiguous()
    kw = dict(scale_value=1.0 / 24.0, query_rope=qr, key_rope=kr, sparse_mode=0)
    ref = module.sparse_flash_attention_grad_triton(q, k, k, idx, do, out, mx, sm, **kw)
    asked = []

    def scarce(nbytes, device):
        asked.append(int(nbytes))
        if len(asked) == 1:
            raise torch.cuda.OutOfMemoryError("no room")
        return _host.workspace(nbytes, device)

    monkeypatch.setattr(module, "workspace", scarce)
    got = module.sparse_flash_attention_grad_triton(q, k, k, idx, do, out, mx, sm, **kw)
    assert len(asked) == 2 and asked[1] == 256 + S2 * (2 * 512 + 64) * 4 < asked[0]
    for n, a, b in zip(NAMES, got, ref):
        sfa_grad_acceptance_rule(host(a), host(b), dtype, name=n, ulps=1.0)


@pytest.mark.parametrize("dtype", ["bf16", "fp16"])
@pytest.mark.parametrize("N1,tensor", [(15, 0), (16, 1), (17, 1)])
@pytest.mark.parametrize("S2", [23, 24, 25, 48, 49])
def test_the_first_tile_and_the_first_head_block(S2, N1, tensor, dtype):
    """The last row sees S2 keys (half of the tcgen05 kernel's softmax warps have none up to 24, a tile is 48), on
    either side of the head count at which that kernel begins; 2 ulp of the io dtype, as everywhere."""
    from dsa_triton_ascend_b200 import _cabi, sparse_flash_attention_grad_triton
    p = _cabi.DsaSfaGradParams()
    p.struct_size = ctypes.sizeof(p)
    for name, kind in p._fields_:
        if kind is ctypes.c_void_p and name not in ("seq_q", "seq_k"):
            setattr(p, name, 256)
    p.batch, p.s1, p.s2, p.n1, p.d, p.d_rope, p.key_rows = 1, 2, S2, N1, 512, 64, S2
    p.sparse_count, p.sparse_block_size, p.sparse_mode = S2, 1, 3
    assert _cabi.lib.dsa_sfa_grad_uses_tensor_path(ctypes.byref(p)) == tensor
    q, k, qr, kr, do = sfa_grad_inputs(S2, 1, 2, S2, N1, 512, 64, dtype)
    idx = sparse_indices(1000 + S2, 1, 2, S2, S2, 1, 3)
    out, mx, sm = sparse_flash_attention_oracle(q, k, idx, qr, kr, 1.0 / 24.0, [2], [S2], sparse_mode=3,
                                                return_softmax_lse=True, dtype=dtype)
    dt = tdtype(dtype)
    tk = dev(k, dt)
    got = sparse_flash_attention_grad_triton(dev(q, dt), tk, tk, dev(idx), dev(do, dt), dev(out, dt), dev(mx), dev(sm),
                                             scale_value=1.0 / 24.0, query_rope=dev(qr, dt), key_rope=dev(kr, dt),
                                             sparse_mode=3)
    ref = sparse_flash_attention_grad_oracle(q, k, idx, do, out, mx, sm, qr, kr, 1.0 / 24.0, [2], [S2], sparse_mode=3,
                                             dtype=dtype)
    for n, a, b in zip(NAMES, got, ref):
        sfa_grad_acceptance_rule(host(a), b, dtype, name=n)
