"""The tcgen05 scoring kernel where its dispatch and its lists of work have edges, against the CUDA-core kernel: few
and odd head counts, paged caches whose block-table look-ups take several rounds, batches that mix row groups of
one and of eight rows."""
import numpy as np
import pytest
import torch

from tests.util import host

pytestmark = pytest.mark.gpu


def _compare(q, k, w, **kw):
    import dsa_triton_ascend_b200.lightning_indexer as li
    out = {}
    for kind in ("tensor", "portable"):
        li.set_kernel(kind)
        try:
            out[kind] = [host(t) for t in li.lightning_indexer_triton(q, k, w, return_value=True, **kw)]
        finally:
            li.set_kernel("auto")
    (ti, tv), (pi, pv) = out["tensor"], out["portable"]
    # as many slots everywhere; values within a rounding step of bf16 (the two kernels add the heads' products in
    # different orders); the same keys except at such boundaries
    assert ((ti >= 0) == (pi >= 0)).all()
    assert np.allclose(tv, pv, rtol=2.0 ** -6, atol=1e-3)
    assert (ti == pi).mean() >= 0.97


def _draw(seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)


def _paged(rng, draw, lens, bs):
    need = [-(-n // bs) for n in lens]
    table = np.full((len(lens), max(need)), -1, np.int32)
    perm, at = rng.permutation(sum(need)), 0
    for b, n in enumerate(need):
        table[b, :n] = perm[at:at + n]
        at += n
    return draw(sum(need), bs, 1, 128), torch.from_numpy(table).cuda()


@pytest.mark.parametrize("heads", [1, 3, 8, 15])
@pytest.mark.parametrize("layout,bs", [("BSND", 0), ("TND", 0), ("PA_BSND", 16), ("PA_BSND", 32), ("PA_BSND", 64),
                                       ("PA_BSND", 128)])
def test_few_heads(heads, layout, bs):
    rng, draw = np.random.RandomState(heads), _draw(heads)
    if layout == "BSND":
        _compare(draw(2, 9, heads, 128), draw(2, 700, 1, 128), draw(2, 9, heads).float(), sparse_count=64)
    elif layout == "TND":
        _compare(draw(14, heads, 128), draw(1500, 1, 128), draw(14, heads).float(), sparse_count=64,
                 layout_query="TND", layout_key="TND", actual_seq_lengths_query=[1, 13, 14],
                 actual_seq_lengths_key=[600, 613, 1500])
    else:
        # (one round of look-ups serves 32 loads: 512 to 4096 keys)
        lens = [5000, 130, 4097]
        k, table = _paged(rng, draw, lens, bs)
        _compare(draw(3, 2, heads, 128), k, draw(3, 2, heads).float(), sparse_count=64, layout_key="PA_BSND",
                 block_table=table, actual_seq_lengths_key=lens)


@pytest.mark.parametrize("rows", [[1] * 20, [1, 1, 60, 1, 3, 1, 9], [70, 8, 33], [1] * 100, [5, 1, 1, 1, 1, 1]])
def test_row_groups_of_mixed_size(rows):
    """TND rows over a paged cache, keys cut into chunks: groups of one to four rows take other chunk sizes than
    groups of five to eight."""
    rng, draw = np.random.RandomState(len(rows)), _draw(sum(rows))
    lens = [int(n) + max(rows) for n in rng.randint(1, 6000, len(rows))]
    k, table = _paged(rng, draw, lens, 128)
    _compare(draw(sum(rows), 64, 128), k, draw(sum(rows), 64).float() / 8, sparse_count=512, layout_query="TND",
             layout_key="PA_BSND", block_table=table, actual_seq_lengths_query=np.cumsum(rows).tolist(),
             actual_seq_lengths_key=lens)
