"""Through the C interface any return_value / return_lse but 0 asks for the results, and 0 leaves the buffers alone; the
`_zeros` entry points store zeros in the place of what is not asked for."""
import ctypes

import pytest
import torch

from dsa_triton_ascend_b200 import _cabi
from dsa_triton_ascend_b200 import lightning_indexer as li


def _filled(p):
    p.struct_size = ctypes.sizeof(p)
    for name, kind in p._fields_:
        if kind is ctypes.c_void_p and name not in ("seq_q", "seq_k", "block_table"):
            setattr(p, name, 256)
    return p


def test_the_zeros_need_somewhere_to_go():
    p = _filled(_cabi.DsaLiParams())
    p.batch, p.s1, p.s2, p.n1, p.n2, p.d, p.sparse_count, p.phases = 1, 4, 16, 8, 1, 128, 8, _cabi.PHASE_ALL
    p.out_values = None
    assert _cabi.lib.dsa_li_forward_zeros(ctypes.byref(p), None, 0, None) == -1
    assert _cabi.lib.dsa_li_forward(ctypes.byref(p), None, 0, None) == -4          # only the workspace is missing
    s = _filled(_cabi.DsaSfaParams())
    s.batch, s.s1, s.s2, s.n1, s.d, s.d_rope, s.sparse_count, s.sparse_block_size, s.key_rows = 1, 4, 16, 8, 512, 64, 8, 1, 16
    for name in ("softmax_max", "softmax_sum"):
        setattr(s, name, None)
        assert _cabi.lib.dsa_sfa_forward_zeros(ctypes.byref(s), None, 0, None) == -1
        assert _cabi.lib.dsa_sfa_forward(ctypes.byref(s), None, 0, None) == -4
        setattr(s, name, 256)


MARK = 7.0


def _index(entry, flag, kernel):
    gen = torch.Generator(device="cuda").manual_seed(3)
    q, k, w = (torch.randn(s, generator=gen, device="cuda").bfloat16() for s in ((1, 9, 16, 128), (1, 300, 1, 128), (1, 9, 16)))
    p, keep, idx, val, _ = li._build_params(q, k, w, None, None, None, "BSND", "BSND", 64, 3, True)
    p.kernel, p.return_value = kernel, flag
    val.fill_(MARK)
    n = ctypes.c_size_t(0)
    assert _cabi.lib.dsa_li_workspace_bytes(ctypes.byref(p), ctypes.byref(n)) == 0
    ws = torch.empty(n.value, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    assert getattr(_cabi.lib, entry)(ctypes.byref(p), ws.data_ptr(), ws.numel(), stream) == 0
    torch.cuda.synchronize()
    return idx.clone(), val.clone()


def _attend(entry, flag, kernel):
    gen = torch.Generator(device="cuda").manual_seed(4)
    rows, keys, heads = 9, 300, 16
    q, qr, k, kr = (torch.randn(s, generator=gen, device="cuda").bfloat16()
                    for s in ((rows, heads, 512), (rows, heads, 64), (keys, 512), (keys, 64)))
    idx = torch.arange(64, dtype=torch.int32, device="cuda").repeat(rows, 1)
    out = torch.empty_like(q)
    mx, sm = (torch.full((rows, heads), MARK, device="cuda") for _ in range(2))
    p = _cabi.DsaSfaParams()
    p.struct_size, p.kernel = ctypes.sizeof(p), kernel
    for name, t in dict(query=q, query_rope=qr, key=k, key_rope=kr, sparse_indices=idx, out=out, softmax_max=mx,
                        softmax_sum=sm).items():
        setattr(p, name, t.data_ptr())
    p.batch, p.s1, p.s2, p.n1, p.d, p.d_rope, p.key_rows = 1, rows, keys, heads, 512, 64, keys
    p.sparse_count, p.sparse_block_size, p.return_lse, p.scale = 64, 1, flag, 1.0 / 24.0
    n = ctypes.c_size_t(0)
    assert _cabi.lib.dsa_sfa_workspace_bytes(ctypes.byref(p), ctypes.byref(n)) == 0
    ws = torch.empty(n.value, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    assert getattr(_cabi.lib, entry)(ctypes.byref(p), ws.data_ptr(), ws.numel(), stream) == 0
    torch.cuda.synchronize()
    return out, torch.stack([mx, sm])


@pytest.mark.gpu
@pytest.mark.parametrize("call,entry", [(_index, "dsa_li_forward"), (_attend, "dsa_sfa_forward")])
@pytest.mark.parametrize("kernel", [_cabi.KERNEL_TENSOR, _cabi.KERNEL_PORTABLE])
def test_any_flag_but_zero_asks_for_the_results(call, entry, kernel):
    main, extra = call(entry, 1, kernel)
    assert not (extra == MARK).any()
    for name in (entry, entry + "_zeros"):
        for flag in (2, -1, 256):
            again = call(name, flag, kernel)
            assert torch.equal(again[0], main) and torch.equal(again[1], extra)
    again = call(entry, 0, kernel)
    assert torch.equal(again[0], main) and (again[1] == MARK).all()
    again = call(entry + "_zeros", 0, kernel)
    assert torch.equal(again[0], main) and not again[1].any()
