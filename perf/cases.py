"""The framework's measured work: calls that a training or serving program makes through the public
operators, over the range of sizes it makes them with.

`listed()` names the fixed cases, `draw(rng)` gives another one of the same ranges, `prepare(case, seed)`
makes what the program holds before the call (inputs on the GPU), `run(state)` is one pass, `work(case)`
the bytes and operations that a pass cannot do without, `tolerance(case)` how far two correct
implementations may be apart.

Kinds of case (`op`):
  index        lightning_indexer alone (prefill)
  attend       sparse_flash_attention alone (prefill)
  prefill      lightning_indexer, its indices straight into sparse_flash_attention (TND)
  decode       the same two calls over paged caches, a few query tokens per sequence
  attend_grad  sparse_flash_attention backward
  sparse_loss  sparse indexer KL loss and its gradients
  dense_loss   softmax statistics of the dense indexer, then the dense KL loss and its gradients
"""
import math

import torch

from dsa_triton_ascend_b200 import (dense_lightning_indexer_softmax_lse_triton, dense_loss_backward_triton,
                                    lightning_indexer_triton, sparse_flash_attention_grad_triton,
                                    sparse_flash_attention_triton, sparse_lightning_indexer_grad_kl_loss_triton)

INDEX_DIM, DIM, ROPE, PAGE = 128, 512, 64, 128
SCALE = 1.0 / math.sqrt(DIM + ROPE)
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # the smallest calls: a short prompt with a narrow indexer / a narrow attention, where what counts
        # is the time from the call to the kernel and the launches
        dict(name="index_short", op="index", layout="BSND", q_lens="512", k_lens="512", heads=8, top_k=64, dtype="bf16"),
        dict(name="attend_short", op="attend", layout="BSND", q_lens="256", k_lens="1024", heads=16, top_k=256,
             dtype="bf16"),
        # prefill of one long prompt: the indexer at its production shape
        dict(name="index_8k", op="index", layout="BSND", q_lens="8192", k_lens="8192", heads=64, top_k=2048,
             dtype="bf16"),
        # prefill of a batch of prompts: the attention at its production shape (the framework's headline)
        dict(name="attend_15k", op="attend", layout="TND", q_lens="8192 4096 2048 1024",
             k_lens="8192 4096 2048 1024", heads=128, top_k=2048, dtype="bf16"),
        # a scheduler's mixed batch: chunks of prompts of odd lengths whose earlier tokens are already
        # cached, a fresh prompt, a lone token; fp16, heads of one of two tensor-parallel ranks
        dict(name="prefill_ragged_fp16", op="prefill", layout="TND", q_lens="377 1029 64 1",
             k_lens="2425 1029 3111 5003", index_heads=64, heads=64, top_k=2048, dtype="fp16"),
        # decode: one token for a few short conversations, and two tokens (one speculated) for a full
        # batch of long ones
        dict(name="decode_8", op="decode", batch=8, q_tokens=1, shortest=2048, longest=12288, index_heads=64,
             heads=128, top_k=2048, dtype="bf16"),
        dict(name="decode_64", op="decode", batch=64, q_tokens=2, shortest=16384, longest=65536, index_heads=64,
             heads=128, top_k=2048, dtype="bf16"),
        # training: the backward operators on a slice of a long context, and on whole packed batches
        dict(name="attend_grad_512", op="attend_grad", layout="BSND", q_lens="512", k_lens="4096", heads=64,
             top_k=2048, dtype="bf16"),
        dict(name="attend_grad_packed", op="attend_grad", layout="TND", q_lens="2048 1361 683",
             k_lens="2048 1361 683", heads=128, top_k=2048, dtype="bf16"),
        dict(name="sparse_loss_512", op="sparse_loss", batch=1, rows=512, keys=4096, heads=64, index_heads=64,
             top_k=2048, dtype="bf16"),
        dict(name="sparse_loss_2k_fp16", op="sparse_loss", batch=1, rows=2048, keys=4096, heads=128, index_heads=64,
             top_k=2048, dtype="fp16"),
        # warm-up stage of the indexer's training: every visible key, multi-head attention keys
        dict(name="dense_loss_512", op="dense_loss", batch=1, rows=512, keys=4096, heads=64, key_heads=64, dim=128,
             index_heads=64, dtype="bf16"),
    ]


# ------------------------------------------------------------------------------------------------
# Drawn cases
# ------------------------------------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _texts(rng, total, cached, most=5):
    """Query and key lengths of a batch of about `total` query tokens; `cached`: keys go back further."""
    parts = [rng.uniform(0.2, 1.0) for _ in range(rng.randint(1, most))]
    q = [max(1, int(total * p / sum(parts))) for p in parts]
    k = [n + (_log_int(rng, 1, cached) if cached and rng.random() < 0.7 else 0) for n in q]
    return " ".join(map(str, q)), " ".join(map(str, k))


def draw(rng):
    most = max(work(c)["flops"] for c in listed() if c["op"] == "attend")
    most_grad = max(work(c)["flops"] for c in listed() if c["op"] == "attend_grad")
    while True:
        op = rng.choice(("index", "attend", "prefill", "decode", "attend_grad", "sparse_loss", "dense_loss"))
        dtype = rng.choice(("bf16", "bf16", "fp16"))
        top_k = rng.choice((64, 256, 512, 1024, 2048, 2048, 2048))
        heads = rng.choice((16, 32, 64, 128))
        index_heads = rng.choice((16, 32, 64, 64))
        if op == "index":
            q, k = _texts(rng, _log_int(rng, 128, 8192), 4096, most=1)
            c = dict(op=op, layout="BSND", q_lens=q, k_lens=k, heads=rng.choice((8, 16, 32, 64, 64)), top_k=top_k,
                     dtype=dtype)
        elif op in ("attend", "attend_grad"):
            layout = rng.choice(("BSND", "TND"))
            total = _log_int(rng, 128, 15360 if op == "attend" else 4096)
            q, k = _texts(rng, total, 4096, most=5 if layout == "TND" else 1)
            c = dict(op=op, layout=layout, q_lens=q, k_lens=k, heads=heads, top_k=top_k, dtype=dtype)
        elif op == "prefill":
            q, k = _texts(rng, _log_int(rng, 128, 8192), 6144)
            c = dict(op=op, layout="TND", q_lens=q, k_lens=k, index_heads=index_heads, heads=heads, top_k=top_k,
                     dtype=dtype)
        elif op == "decode":
            shortest = _log_int(rng, 512, 16384)
            c = dict(op=op, batch=_log_int(rng, 1, 64), q_tokens=rng.choice((1, 1, 2)), shortest=shortest,
                     longest=rng.randint(shortest, 4 * shortest), index_heads=index_heads, heads=heads, top_k=top_k,
                     dtype=dtype)
        elif op == "sparse_loss":
            rows = _log_int(rng, 64, 2048)
            c = dict(op=op, batch=rng.choice((1, 1, 2)), rows=rows, keys=rows + max(top_k, _log_int(rng, 64, 4096)),
                     heads=heads, index_heads=index_heads, top_k=top_k, dtype=dtype)
        else:
            rows = _log_int(rng, 64, 1024)
            many = rng.random() < 0.7
            c = dict(op=op, batch=rng.choice((1, 1, 2)), rows=rows, keys=rows + _log_int(rng, 64, 4096),
                     heads=heads, key_heads=heads if many else 1, dim=128 if many else 512, index_heads=index_heads,
                     dtype=dtype)
        if work(c)["flops"] <= (most if op in ("index", "attend", "prefill", "decode") else most_grad / 4 if
                                op == "dense_loss" else most_grad):
            return c


# ------------------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------------------
def _ints(text):
    return [int(v) for v in text.split()]


def _ends(lens):
    out, at = [], 0
    for n in lens:
        at += n
        out.append(at)
    return out


def _visible(q_len, k_len):
    """Keys that each of the q_len query tokens sees under the right-down causal mask."""
    return [max(0, k_len - q_len + i + 1) for i in range(q_len)]


class _Draws:
    """Seeded normal tensors on the GPU, made in pieces so that the fp32 staging stays small."""

    def __init__(self, seed, dtype):
        self.gen, self.dtype = torch.Generator(device="cuda").manual_seed(seed), DTYPES[dtype]

    def normal(self, *shape, scale=1.0, dtype=None):
        out = torch.empty(shape, dtype=dtype or self.dtype, device="cuda")
        flat = out.view(-1)
        for i in range(0, flat.numel(), 1 << 26):
            n = min(1 << 26, flat.numel() - i)
            flat[i:i + n] = torch.randn(n, generator=self.gen, device="cuda") * scale
        return out

    def selection(self, q_len, k_len, top_k):
        """[q_len, top_k]: distinct visible keys of each row in random order, -1 past the visible ones."""
        out = torch.full((q_len, top_k), -1, dtype=torch.int32, device="cuda")
        n = min(top_k, k_len)
        for i in range(0, q_len, 2048):
            m = min(2048, q_len - i)
            visible = k_len - q_len + i + 1 + torch.arange(m, device="cuda")
            score = torch.rand(m, k_len, generator=self.gen, device="cuda")
            score.masked_fill_(torch.arange(k_len, device="cuda")[None, :] >= visible[:, None], -1.0)
            best = torch.topk(score, n, dim=1)
            out[i:i + m, :n] = torch.where(best.values >= 0, best.indices, -1).to(torch.int32)
        return out


def _forward_state(q, k, qr, kr, idx):
    """Output and softmax statistics of the attention over the selected keys: one sequence,
    q [S1,N1,D], k [S2,D], idx [S1,K] -> out in q's dtype, max and sum fp32 [S1,N1]."""
    out = torch.empty_like(q)
    mx = torch.empty(q.shape[:2], dtype=torch.float32, device="cuda")
    sm = torch.empty_like(mx)
    step = max(1, (1 << 27) // (idx.shape[1] * (k.shape[1] + kr.shape[1])))
    for i in range(0, q.shape[0], step):
        s = slice(i, i + step)
        sel = idx[s].long()
        kk = k[sel.clamp_min(0)]
        x = (torch.bmm(q[s], kk.transpose(1, 2)).float() +
             torch.bmm(qr[s], kr[sel.clamp_min(0)].transpose(1, 2)).float()) * SCALE
        x.masked_fill_((sel < 0)[:, None, :], -math.inf)
        mx[s] = x.amax(-1)
        x = (x - mx[s][..., None]).exp_()
        sm[s] = x.sum(-1)
        out[s] = torch.bmm((x / sm[s][..., None]).to(q.dtype), kk)
    return out, mx, sm


def _dense_statistics(q, k, qr, kr, scale):
    """Softmax maximum and sum over all visible keys: q [B,S1,N1,D], k [B,S2,N2,D] -> [B,N2,S1,N1/N2]."""
    B, S1, N1, _ = q.shape
    S2, N2 = k.shape[1], k.shape[2]
    mx = torch.empty(B, N2, S1, N1 // N2, dtype=torch.float32, device="cuda")
    sm = torch.empty_like(mx)
    hidden = torch.arange(S2, device="cuda")[None, :] > (S2 - S1 + torch.arange(S1, device="cuda"))[:, None]
    for b in range(B):
        for h in range(N1):
            kh = h // (N1 // N2)
            x = (q[b, :, h] @ k[b, :, kh].T).float() + (qr[b, :, h] @ kr[b, :, kh].T).float()
            x = (x * scale).masked_fill_(hidden, -math.inf)
            top = x.amax(-1)
            mx[b, kh, :, h % (N1 // N2)] = top
            sm[b, kh, :, h % (N1 // N2)] = (x - top[:, None]).exp_().sum(-1)
    return mx, sm


def prepare(case, seed):
    d = _Draws(seed, case["dtype"])
    c = dict(case)
    op = c["op"]
    if op in ("index", "attend", "prefill", "attend_grad"):
        ql, kl = _ints(c["q_lens"]), _ints(c["k_lens"])
        tnd = c["layout"] == "TND"
        lead_q = (sum(ql),) if tnd else (1, ql[0])
        lead_k = (sum(kl),) if tnd else (1, kl[0])
        s = dict(op=op, layout=c["layout"], top_k=c["top_k"], ends_q=_ends(ql) if tnd else None,
                 ends_k=_ends(kl) if tnd else None)
        if op in ("index", "prefill"):
            heads = c["heads"] if op == "index" else c["index_heads"]
            s.update(qi=d.normal(*lead_q, heads, INDEX_DIM), ki=d.normal(*lead_k, 1, INDEX_DIM),
                     w=d.normal(*lead_q, heads, scale=1 / math.sqrt(heads), dtype=torch.float32))
        if op != "index":
            scale = 0.3 if op == "attend_grad" else 1.0
            s.update(q=d.normal(*lead_q, c["heads"], DIM, scale=scale), k=d.normal(*lead_k, 1, DIM, scale=scale),
                     qr=d.normal(*lead_q, c["heads"], ROPE, scale=scale), kr=d.normal(*lead_k, 1, ROPE, scale=scale))
        if op in ("attend", "attend_grad"):
            idx = [d.selection(a, b, c["top_k"]) for a, b in zip(ql, kl)]
            s["idx"] = torch.cat(idx).view(*lead_q, 1, c["top_k"])
        if op == "attend_grad":
            s["d_out"] = d.normal(*lead_q, c["heads"], DIM, scale=0.3)
            flat = [s[n].view(-1, *s[n].shape[-2:]) for n in ("q", "qr")] + \
                   [s[n].view(-1, s[n].shape[-1]) for n in ("k", "kr")]
            parts, tq, tk = [], 0, 0
            for a, b, i in zip(ql, kl, idx):
                parts.append(_forward_state(flat[0][tq:tq + a], flat[2][tk:tk + b], flat[1][tq:tq + a],
                                            flat[3][tk:tk + b], i))
                tq, tk = tq + a, tk + b
            out, mx, sm = (torch.cat(p) for p in zip(*parts))
            stat = (1, sum(ql), c["heads"]) if tnd else (1, 1, ql[0], c["heads"])
            s.update(out=out.view_as(s["q"]), mx=mx.view(stat), sm=sm.view(stat))
        return s
    if op == "decode":
        B, S1 = c["batch"], c["q_tokens"]
        lens = torch.randint(c["shortest"], c["longest"] + 1, (B,), generator=d.gen, device="cuda", dtype=torch.int32)
        need = (-(-lens // PAGE)).tolist()
        # the table is as wide as the longest sequence may get; pages are handed out in random order
        width = -(-c["longest"] // PAGE)
        pages = torch.randperm(sum(need), generator=d.gen, device="cuda").to(torch.int32)
        table = torch.full((B, width), -1, dtype=torch.int32, device="cuda")
        for b, part in enumerate(pages.split(need)):
            table[b, :need[b]] = part
        return dict(op=op, top_k=c["top_k"], lens=lens, table=table, qi=d.normal(B, S1, c["index_heads"], INDEX_DIM),
                    ki=d.normal(sum(need), PAGE, 1, INDEX_DIM),
                    w=d.normal(B, S1, c["index_heads"], scale=1 / math.sqrt(c["index_heads"]), dtype=torch.float32),
                    q=d.normal(B, S1, c["heads"], DIM), qr=d.normal(B, S1, c["heads"], ROPE),
                    k=d.normal(sum(need), PAGE, 1, DIM), kr=d.normal(sum(need), PAGE, 1, ROPE))
    B, S1, S2, N1, G = c["batch"], c["rows"], c["keys"], c["heads"], c["index_heads"]
    N2, D = c.get("key_heads", 1), c.get("dim", DIM)
    s = dict(op=op, scale=1.0 / math.sqrt(D + ROPE), q=d.normal(B, S1, N1, D, scale=0.3),
             k=d.normal(B, S2, N2, D, scale=0.3), qr=d.normal(B, S1, N1, ROPE, scale=0.3),
             kr=d.normal(B, S2, N2, ROPE, scale=0.3), qi=d.normal(B, S1, G, INDEX_DIM, scale=0.3),
             ki=d.normal(B, S2, 1, INDEX_DIM, scale=0.3), w=d.normal(B, S1, G, scale=0.3).abs_())
    s["mx"], s["sm"] = _dense_statistics(s["q"], s["k"], s["qr"], s["kr"], s["scale"])
    if op == "sparse_loss":
        s["idx"] = torch.stack([d.selection(S1, S2, c["top_k"]) for _ in range(B)]).view(B, S1, 1, c["top_k"])
    return s


# ------------------------------------------------------------------------------------------------
# One pass
# ------------------------------------------------------------------------------------------------
def run(s):
    op = s["op"]
    if op in ("index", "prefill"):
        idx, values = lightning_indexer_triton(
            s["qi"], s["ki"], s["w"], actual_seq_lengths_query=s["ends_q"], actual_seq_lengths_key=s["ends_k"],
            layout_query=s["layout"], layout_key=s["layout"], sparse_count=s["top_k"], sparse_mode=3)
        if op == "index":
            return idx, values
    if op in ("attend", "prefill"):
        attended = sparse_flash_attention_triton(
            s["q"], s["k"], s["k"], s["idx"] if op == "attend" else idx, scale_value=SCALE,
            actual_seq_lengths_query=s["ends_q"], actual_seq_lengths_kv=s["ends_k"], query_rope=s["qr"],
            key_rope=s["kr"], layout_query=s["layout"], layout_kv=s["layout"], sparse_mode=3, return_softmax_lse=True)
        return attended if op == "attend" else (idx,) + attended
    if op == "decode":
        idx, _ = lightning_indexer_triton(
            s["qi"], s["ki"], s["w"], actual_seq_lengths_key=s["lens"], block_table=s["table"],
            layout_key="PA_BSND", sparse_count=s["top_k"], sparse_mode=3)
        return (idx,) + sparse_flash_attention_triton(
            s["q"], s["k"], s["k"], idx, scale_value=SCALE, block_table=s["table"], actual_seq_lengths_kv=s["lens"],
            query_rope=s["qr"], key_rope=s["kr"], layout_kv="PA_BSND", sparse_mode=3, block_size=PAGE)
    if op == "attend_grad":
        return sparse_flash_attention_grad_triton(
            s["q"], s["k"], s["k"], s["idx"], s["d_out"], s["out"], s["mx"], s["sm"], scale_value=SCALE,
            query_rope=s["qr"], key_rope=s["kr"], actual_seq_lengths_query=s["ends_q"],
            actual_seq_lengths_kv=s["ends_k"], layout=s["layout"], sparse_mode=3)
    if op == "sparse_loss":
        return sparse_lightning_indexer_grad_kl_loss_triton(
            s["q"], s["k"], s["qi"], s["ki"], s["w"], s["idx"], s["mx"], s["sm"], query_rope=s["qr"],
            key_rope=s["kr"], scale_value=s["scale"])
    top, total = dense_lightning_indexer_softmax_lse_triton(s["qi"], s["ki"], s["w"])
    return (top, total) + dense_loss_backward_triton(
        s["q"], s["k"], s["qi"], s["ki"], s["w"], s["mx"], s["sm"], top, total, s["scale"], query_rope=s["qr"],
        key_rope=s["kr"])


# ------------------------------------------------------------------------------------------------
# What a pass cannot do without
# ------------------------------------------------------------------------------------------------
def work(case):
    c, op = case, case["op"]
    if op in ("index", "attend", "prefill", "attend_grad"):
        ql, kl, k = _ints(c["q_lens"]), _ints(c["k_lens"]), c["top_k"]
        seen = [v for a, b in zip(ql, kl) for v in _visible(a, b)]
    elif op == "decode":
        mean = (c["shortest"] + c["longest"]) // 2
        ql, kl, k = [c["q_tokens"]] * c["batch"], [mean] * c["batch"], c["top_k"]
        seen = [mean] * (c["batch"] * c["q_tokens"])
    else:
        ql, kl, k = [c["rows"]] * c["batch"], [c["keys"]] * c["batch"], c.get("top_k", c["keys"])
        seen = [v for a, b in zip(ql, kl) for v in _visible(a, b)]
    tokens, keys, pairs = sum(ql), sum(kl), sum(seen)
    chosen = sum(min(k, v) for v in seen)
    heads, index_heads = c["heads"], c["heads"] if op == "index" else c.get("index_heads", 0)
    # indexer: queries, weights and keys in, indices (and the zeros of unused values) out
    index_bytes = 2 * INDEX_DIM * (tokens * index_heads + keys) + 4 * tokens * index_heads + 6 * tokens * k
    index_flops = 2.0 * pairs * index_heads * INDEX_DIM
    # attention: queries, indices and the keys that the indices can reach in, output and statistics out
    reached = sum(min(b, a * k) for a, b in zip(ql, kl))
    attend_bytes = 2 * (DIM + ROPE) * (tokens * heads + reached) + 4 * tokens * k + 2 * DIM * tokens * heads + \
        8 * tokens * heads
    attend_flops = 2.0 * chosen * heads * (2 * DIM + ROPE)
    if op == "index":
        return dict(bytes=index_bytes, flops=index_flops)
    if op == "attend":
        return dict(bytes=attend_bytes, flops=attend_flops)
    if op in ("prefill", "decode"):
        return dict(bytes=index_bytes + attend_bytes, flops=index_flops + attend_flops)
    if op == "attend_grad":   # q, k, dO, O, indices, statistics in; dQ, dK, dV out; five contractions
        return dict(bytes=2 * tokens * heads * (2 * (DIM + ROPE) + 2 * DIM) + 2 * keys * (2 * (DIM + ROPE) + DIM) +
                    4 * tokens * k + 8 * tokens * heads,
                    flops=2.0 * chosen * heads * (3 * (DIM + ROPE) + 2 * DIM))
    D, N2 = c.get("dim", DIM), c.get("key_heads", 1)
    used = chosen if op == "sparse_loss" else pairs
    loss_bytes = 2 * (D + ROPE) * (tokens * heads + keys * N2) + 4 * INDEX_DIM * (tokens * index_heads + keys) + \
        4 * tokens * index_heads + 8 * tokens * heads + (4 * tokens * k if op == "sparse_loss" else 16 * tokens)
    # attention probabilities; index scores, d_weights with them; d_query_index; d_key_index
    loss_flops = 2.0 * used * (heads * (D + ROPE) + 3 * index_heads * INDEX_DIM)
    return dict(bytes=loss_bytes, flops=loss_flops)


def tolerance(case):
    """Outputs leave in 16 bits (or are fp32 sums of products of probabilities rounded to 16 bits): one
    rounding is 2^-9 of the value for bf16, 2^-12 for fp16, intermediate probabilities and score gradients
    are rounded the same way.  Indices are ranked by scores rounded to 16 bits: a sum taken in another order
    (1e-6 relative) moves about one score in 3000 over a rounding boundary and with it its neighbours among
    the equals."""
    rel = 1e-2 if case["dtype"] == "bf16" else 4e-3
    if case["op"] in ("index", "prefill", "decode"):
        return {"rel": rel, "differ": 0.005}
    return {"rel": rel}
