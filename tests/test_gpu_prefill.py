"""-m gpu parity tests for the tcgen05 varlen prefill attention (K3 dense, K4 paged prefix) vs the CPU oracle."""
import os

import numpy as np
import pytest
import torch

from oracle import layers as O
from tests.util import assert_close, cache_to_layout, make_paged_kv, randn_bf16, to_dev_bf16, to_np_f32

pytestmark = pytest.mark.gpu
ATT_ATOL, ATT_RTOL = 1e-2, 1.6e-2   # attention tolerance (2 bf16 ulps of the output + P rounding)


def _cu(lens):
    return np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)


DENSE = [
    ([1], 4, 2), ([5], 16, 8), ([64], 4, 4), ([65, 1, 128], 4, 2), ([129, 256, 257], 8, 2), ([300, 513, 7], 16, 8),
    ([1024], 32, 8), ([128] * 4, 16, 8),   # the last one is the 4 x 128-token prefill of Qwen3-0.6B
]


@pytest.mark.parametrize("lens,H,Hkv", DENSE, ids=[str(i) for i in range(len(DENSE))])
def test_varlen_prefill_dense_vs_oracle(cuda, lens, H, Hkv):
    from nano_vllm_rs_b200 import ops
    D = 128
    rng = np.random.default_rng(sum(lens) + H)
    n = sum(lens)
    # q/k/v as column slices of one packed qkv buffer (how the model calls it: strided rows)
    qkv = randn_bf16(rng, (n, (H + 2 * Hkv) * D))
    q = qkv[:, : H * D].reshape(n, H, D); k = qkv[:, H * D : (H + Hkv) * D].reshape(n, Hkv, D)
    v = qkv[:, (H + Hkv) * D :].reshape(n, Hkv, D)
    cu = _cu(lens)
    scale = 1 / np.sqrt(D)
    ref = O.flash_attention_varlen(q, k, v, cu, cu, scale)
    t = to_dev_bf16(qkv, cuda)
    qd = t[:, : H * D].view(n, H, D); kd = t[:, H * D : (H + Hkv) * D].view(n, Hkv, D); vd = t[:, (H + Hkv) * D :].view(n, Hkv, D)
    cud = torch.from_numpy(cu).to(cuda)
    out = ops.varlen_prefill_attention(qd, kd, vd, cud, cud, max(lens), max(lens), scale=scale)
    torch.cuda.synchronize()
    assert_close(to_np_f32(out), ref, ATT_ATOL, ATT_RTOL, f"prefill dense {lens}")


PAGED = [
    # (prefix_lens, suffix_lens, H, Hkv, block_size)
    ([256], [44], 4, 2, 256), ([0, 512, 256], [300, 1, 129], 16, 8, 256), ([64, 128], [16, 70], 4, 2, 64),
    ([32, 0, 48], [17, 33, 100], 4, 1, 16), ([4096], [256], 8, 8, 256),
]


@pytest.mark.parametrize("kind", ["reference", "head_major"])
@pytest.mark.parametrize("case", PAGED, ids=[str(i) for i in range(len(PAGED))])
def test_varlen_prefill_paged_prefix_vs_oracle(cuda, kind, case):
    """flash_attention_varlen_with_cache (attention.rs:211-222 intent): the suffix queries attend to prefix + suffix
    read back from the paged cache (all K/V of the step already stored — note N2)."""
    from nano_vllm_rs_b200 import ops
    from nano_vllm_rs_b200._ffi import KvLayout
    pre, suf, H, Hkv, bs = case
    D = 128
    rng = np.random.default_rng(sum(pre) + sum(suf) + bs)
    tot = [a + b for a, b in zip(pre, suf)]
    kc, vc, tables, ks, vs = make_paged_kv(rng, tot, bs, Hkv, D)
    nq = sum(suf)
    q = randn_bf16(rng, (nq, H, D))
    cu_q, cu_k = _cu(suf), _cu(tot)
    scale = 1 / np.sqrt(D)
    ref = O.flash_attention_varlen_with_cache(q, kc, vc, tables, cu_q, cu_k, scale)
    lay = KvLayout.reference(bs, Hkv, D) if kind == "reference" else KvLayout.head_major(bs, Hkv, D)
    out = ops.varlen_prefill_attention(to_dev_bf16(q, cuda), None, None, torch.from_numpy(cu_q).to(cuda),
                                       torch.from_numpy(cu_k).to(cuda), max(suf), max(tot), scale=scale,
                                       k_cache=cache_to_layout(kc, kind, cuda), v_cache=cache_to_layout(vc, kind, cuda),
                                       block_tables=torch.from_numpy(tables).to(cuda), layout=lay)
    torch.cuda.synchronize()
    assert_close(to_np_f32(out), ref, ATT_ATOL, ATT_RTOL, f"prefill paged {case}")


def test_varlen_prefill_full_size_vs_torch(cuda):
    """A full prefill step: 64 seqs x 512 tokens, 16/8 heads — against torch SDPA (fp32 math on the
    device) on sampled sequences, plus the paged == dense consistency property."""
    from nano_vllm_rs_b200 import ops
    B, L, H, Hkv, D = 64, 512, 16, 8, 128
    g = torch.Generator(device="cuda").manual_seed(3)
    q = torch.randn((B * L, H, D), generator=g, device=cuda).to(torch.bfloat16)
    k = torch.randn((B * L, Hkv, D), generator=g, device=cuda).to(torch.bfloat16)
    v = torch.randn((B * L, Hkv, D), generator=g, device=cuda).to(torch.bfloat16)
    cu = torch.arange(0, B * L + 1, L, dtype=torch.int32, device=cuda)
    out = ops.varlen_prefill_attention(q, k, v, cu, cu, L, L)
    torch.cuda.synchronize()
    for b in (0, 17, 63):
        sl = slice(b * L, (b + 1) * L)
        qq = q[sl].float().permute(1, 0, 2); kk = k[sl].float().permute(1, 0, 2).repeat_interleave(H // Hkv, 0)
        vv = v[sl].float().permute(1, 0, 2).repeat_interleave(H // Hkv, 0)
        ref = torch.nn.functional.scaled_dot_product_attention(qq, kk, vv, is_causal=True).permute(1, 0, 2)
        assert_close(to_np_f32(out[sl]), to_np_f32(ref), ATT_ATOL, ATT_RTOL, f"prefill full-size seq {b}")


@pytest.mark.parametrize("H,Hkv,top,paged", [(16, 8, 700, 0), (6, 2, 500, 0), (8, 8, 300, 0), (16, 8, 300, 64), (6, 2, 200, 256), (8, 2, 130, 16)])
def test_varlen_prefill_many_ragged_items(cuda, H, Hkv, top, paged):
    """More work items than SMs, most of them claimed by CTAs that stay, many of them empty: 60 sequences of 0 .. top new tokens (heads that pair
    up and heads that do not, tiles of one to a dozen), dense and behind a paged prefix, against torch in f32."""
    from nano_vllm_rs_b200 import ops
    from nano_vllm_rs_b200._ffi import KvLayout
    D, B = 128, 60
    rng = np.random.default_rng(H + top)
    lens = [int(top * u * u) for u in rng.random(B)]
    lens[5], lens[17], lens[40] = 0, top, 1
    pre = [int(rng.integers(0, 300)) if paged else 0 for _ in lens]
    tot = [a + b for a, b in zip(pre, lens)]
    g = torch.Generator(device="cuda").manual_seed(top)
    rand = lambda *s: torch.randn(*s, generator=g, device=cuda).to(torch.bfloat16)
    q = rand(sum(lens), H, D)
    ks, vs = [rand(n, Hkv, D) for n in tot], [rand(n, Hkv, D) for n in tot]
    cu_q, cu_k = torch.from_numpy(_cu(lens)).to(cuda), torch.from_numpy(_cu(tot)).to(cuda)
    if not paged:
        out = ops.varlen_prefill_attention(q, torch.cat(ks), torch.cat(vs), cu_q, cu_k, max(lens), max(tot))
    else:
        per = [-(-n // paged) for n in tot]
        ids = iter(torch.randperm(sum(per), generator=torch.Generator().manual_seed(1)).tolist())
        tables = torch.full((B, max(per)), -1, dtype=torch.int32)
        kc, vc = (torch.zeros(sum(per), Hkv, paged, D, dtype=torch.bfloat16, device=cuda) for _ in range(2))
        for b in range(B):
            for i in range(per[b]):
                blk = next(ids)
                tables[b, i] = blk
                n = min(paged, tot[b] - i * paged)
                kc[blk, :, :n] = ks[b][i * paged:i * paged + n].transpose(0, 1)
                vc[blk, :, :n] = vs[b][i * paged:i * paged + n].transpose(0, 1)
        out = ops.varlen_prefill_attention(q, None, None, cu_q, cu_k, max(lens), max(tot), k_cache=kc, v_cache=vc, block_tables=tables.to(cuda),
                                           layout=KvLayout.head_major(paged, Hkv, D))
    torch.cuda.synchronize()
    at = 0
    for b, n in enumerate(lens):
        if n:
            s = torch.einsum("qhd,khd->hqk", q[at:at + n].float(), ks[b].float().repeat_interleave(H // Hkv, 1)) * D ** -0.5
            hidden = torch.arange(tot[b], device=cuda)[None, :] > torch.arange(n, device=cuda)[:, None] + pre[b]
            ref = torch.einsum("hqk,khd->qhd", s.masked_fill(hidden, -float("inf")).softmax(-1), vs[b].float().repeat_interleave(H // Hkv, 1))
            assert_close(to_np_f32(out[at:at + n]), to_np_f32(ref), ATT_ATOL, ATT_RTOL, f"sequence {b}: {n} of {tot[b]}")
        at += n


@pytest.mark.parametrize("paged", [False, True])
@pytest.mark.parametrize("H,Hkv", [(4, 2), (3, 3)])
def test_no_number_reaches_only_the_tokens_that_see_it(cuda, H, Hkv, paged):
    """NaN in the second sequence's keys and values, in one value in the middle of the first, and behind its last token in its block: rows that see
    none of them are what they are without them."""
    from nano_vllm_rs_b200 import ops
    from nano_vllm_rs_b200._ffi import KvLayout
    D, bs, lens, mid = 128, 256, [300, 200], 170
    rng = np.random.default_rng(3)
    kc, vc, tables, ks, vs = make_paged_kv(rng, lens, bs, Hkv, D)
    cu = torch.from_numpy(_cu(lens)).to(cuda)
    q = to_dev_bf16(randn_bf16(rng, (sum(lens), H, D)), cuda)
    if paged:
        kd, vd = (cache_to_layout(x, "reference", cuda) for x in (kc, vc))
        flat = lambda x: x.view(-1, Hkv, D)
        row = lambda s, j: int(tables[s, j // bs]) * bs + j % bs
        call = lambda: ops.varlen_prefill_attention(q, None, None, cu, cu, max(lens), max(lens), k_cache=kd, v_cache=vd,
                                                    block_tables=torch.from_numpy(tables).to(cuda), layout=KvLayout.reference(bs, Hkv, D))
    else:
        kd, vd = (to_dev_bf16(np.concatenate(x), cuda) for x in (ks, vs))
        flat = lambda x: x
        row = lambda s, j: sum(lens[:s]) + j
        call = lambda: ops.varlen_prefill_attention(q, kd, vd, cu, cu, max(lens), max(lens))
    clean = call()
    for j in range(lens[1]): flat(kd)[row(1, j)], flat(vd)[row(1, j)] = float("nan"), float("nan")
    flat(vd)[row(0, mid), 0, 5] = float("nan")
    if paged:
        for j in range(lens[0], -(-lens[0] // bs) * bs): flat(kd)[row(0, j)], flat(vd)[row(0, j)] = float("nan"), float("inf")
    out = call()
    torch.cuda.synchronize()
    hit = torch.zeros_like(out, dtype=torch.bool)
    hit[mid:lens[0], :H // Hkv, 5] = True
    hit[lens[0]:] = True
    assert torch.equal(torch.isnan(out), hit)
    assert_close(to_np_f32(out[~hit]), to_np_f32(clean[~hit]), ATT_ATOL, ATT_RTOL, "rows that do not see it")
