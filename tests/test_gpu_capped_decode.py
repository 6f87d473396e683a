"""Attention of single tokens with heads of 128 values (capped_decode.cu) against 64 bits, where its tiles, shares and options can go wrong."""
import math

import numpy as np
import pytest
import torch

from tests.arch_util import paged

D = 128


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv,bs,window,softcap,extra,cap", [
    (4, 4, 16, 0, 0.0, "", 0), (16, 4, 256, 0, 50.0, "gate temp", 64), (11, 1, 48, 0, 0.0, "sinks headgate", 64), (16, 2, 32, 70, 0.0, "", 64),
    (32, 2, 64, 33, 5.0, "sinks gate", 0), (6, 2, 16, 1000, 0.0, "temp", 300)])
def test_single_tokens_at_the_edges_of_tiles(cuda, heads, kv, bs, window, softcap, extra, cap):
    """Contexts around sub-tiles (16 keys), tiles (64) and shares; `cap` extra blocks in the tables let clusters share the keys.  Rows that a
    token does not see hold NaN: none may reach it.  Two tokens of one sequence beside a sequence without any: as many tokens as sequences.
    Tolerance: P and the output are rounded to bf16, which is off by 2^-8 at the most and about 1.7e-3 in the mean square, each; the rest
    is f32.  2.4e-3 together, with room for rows of few keys, whose roundings of P do not average out."""
    from nano_vllm_rs_b200 import ops
    ctx = [1, 15, 16, 17, 31, 63, 64, 65, 127, 128, 129, 193, 257, 300, 513, 1025]
    rng, gen = np.random.default_rng(heads), torch.Generator(device="cuda").manual_seed(heads)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    seqs, pos = list(range(len(ctx))) + [len(ctx) - 1], [c - 1 for c in ctx] + [1025]     # the last sequence has two tokens, the 17th none
    ctx[-1] = 1026
    tables, _, nslots = paged(rng, ctx + [5], bs)
    if cap:
        tables = np.concatenate([tables, np.full((len(ctx) + 1, cap), -1, np.int32)], 1)
    tabs = torch.from_numpy(tables).cuda()
    kc, vc = (torch.full((nslots, kv * D + 8), math.nan, device="cuda", dtype=torch.bfloat16) for _ in "kv")
    at = lambda s, j: tabs[s].long()[j // bs] * bs + j % bs
    for s, c in enumerate(ctx):
        first = min(p for t, p in zip(seqs, pos) if t == s)
        rows = at(s, torch.arange(max(0, first + 1 - window) if window else 0, c, device="cuda"))
        kc[rows], vc[rows] = randn(len(rows), kv * D + 8).to(torch.bfloat16), randn(len(rows), kv * D + 8).to(torch.bfloat16)
    n, g = len(seqs), heads // kv
    q = randn(n, heads * D).to(torch.bfloat16)
    gate = randn(n, heads * D) if " gate" in " " + extra else (randn(n, heads) if "headgate" in extra else None)
    sinks = randn(heads) if "sinks" in extra else None
    coef, every, scale = (0.3, 16, 0.1) if "temp" in extra else (0.0, 1, 0.1)
    cu = torch.tensor([0] + [sum(t < i for t in seqs) for i in range(1, len(ctx) + 2)], device="cuda", dtype=torch.int32)
    assert cu.shape[0] - 1 == n and int(cu[-1]) == n
    out = ops.window_attention(q, gate, kc, vc, torch.tensor(seqs, device="cuda", dtype=torch.int32), torch.tensor(pos, device="cuda"), tabs, bs, heads, kv, D, D, scale, window,
                               sinks, "headgate" in extra, softcap, coef, every, cu)
    for t in range(n):
        rows = at(seqs[t], torch.arange(max(0, pos[t] + 1 - window) if window else 0, pos[t] + 1, device="cuda"))
        k, v = (c[rows][:, :kv * D].double().reshape(-1, kv, D).repeat_interleave(g, 1) for c in (kc, vc))
        s = torch.einsum("hd,jhd->hj", q[t].double().reshape(heads, D), k) * scale * (1 + coef * math.log((pos[t] + 1) // every + 1))
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        if sinks is not None:
            s = torch.cat([s, sinks.double()[:, None]], 1)
        ref = torch.einsum("hj,jhd->hd", torch.softmax(s, -1)[:, :len(rows)], v)
        if gate is not None:
            ref = ref * torch.sigmoid(gate[t].double().reshape(heads, -1))
        err = out[t].double().reshape(heads, D) - ref
        assert float(err.norm() / ref.norm()) < 6e-3, (t, pos[t])


@pytest.mark.gpu
@pytest.mark.parametrize("offset,pad", [(2, 6), (0, 2), (1, 7)])
def test_queries_off_16_bytes_keep_their_probabilities_in_f32(cuda, offset, pad):
    """Two keys of weights 1 and 1 - 2^-10 whose values cancel: what is left, 2^-11, is gone where the weights are rounded to bf16.  Tolerance: the output's own
    rounding, 2^-9, and a key's value in bf16 (2^-9 of a score of 2^-10)."""
    from nano_vllm_rs_b200 import ops
    heads, kv, bs, n = 4, 2, 16, 2
    kc, vc = (torch.zeros(4 * bs, kv * D, device="cuda", dtype=torch.bfloat16) for _ in "kv")
    tabs = torch.tensor([[2, -1], [1, -1]], device="cuda", dtype=torch.int32)
    for b in (1, 2):
        kc[b * bs + 1, ::D] = -(2.0 ** -10)
        vc[b * bs], vc[b * bs + 1] = 1.0, -1.0
    q = torch.zeros(n, heads * D + pad + offset, device="cuda", dtype=torch.bfloat16)[:, offset:offset + heads * D]
    q[:, ::D] = 1.0
    out = ops.window_attention(q, None, kc, vc, torch.arange(n, device="cuda", dtype=torch.int32), torch.ones(n, device="cuda", dtype=torch.int64), tabs, bs, heads, kv, D, D, 1.0,
                               cu_tokens=torch.arange(n + 1, device="cuda", dtype=torch.int32))
    p = math.exp(-(2.0 ** -10))
    assert ((out.double() / ((1 - p) / (1 + p)) - 1).abs() < 5e-3).all()
