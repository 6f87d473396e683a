"""Latent attention of single tokens with kv_rank 512 (latent_attn_decode.cu) against 64 bits, where its tiles, shares and copies can go wrong."""
import math

import numpy as np
import pytest
import torch

from tests.arch_util import paged

RANK = 512


def attend(q_abs, q, seq, pos, tabs, bs, cache, heads, dim, rot, scale, window=0, sinks=None, gate=None):
    from nano_vllm_rs_b200 import _ffi
    n = q_abs.shape[0]
    out = torch.full((n, heads * RANK), 7.0, dtype=torch.bfloat16, device="cuda")
    p = lambda t: t.data_ptr() if t is not None else None
    _ffi.check(_ffi.lib().nvllm_latent_step_attention(p(out), out.stride(0), p(q_abs), q_abs.stride(0), p(q), q.stride(0), p(seq), p(pos), p(tabs), tabs.shape[1],
                                                      bs, p(cache), cache.stride(0), n, n, heads, dim, rot, RANK, scale, window, p(sinks), p(gate), heads, None,
                                                      0, 0, torch.cuda.current_stream().cuda_stream))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("heads,rot,bs,window,cap", [
    (16, 64, 256, 0, 0), (16, 64, 48, 0, 64), (3, 0, 16, 40, 0), (33, 6, 32, 0, 64), (16, 8, 256, 33, 64), (5, 62, 8, 1000, 64)])
def test_single_tokens_at_the_edges_of_tiles(cuda, heads, rot, bs, window, cap):
    """Contexts around multiples of the 32-key tile and of the ring; `cap` extra blocks in the tables let clusters share the keys.  Rows that
    a token does not see (behind its context, before its window) hold NaN: none may reach it.  Tolerance: P and the output are rounded to
    bf16, which is off by 2^-8 at the most and about 1.7e-3 in the mean square, each; the rest is f32.  2.4e-3 together, with room for rows of
    few keys, whose roundings of P do not average out."""
    ctx = [1, 2, 31, 32, 33, 63, 64, 65, 127, 129, 160, 161, 193, 320, 385, 700, 1025]
    n, dim, scale, row = len(ctx), 10, 0.25, -(-(RANK + rot) // 8) * 8
    rng, gen = np.random.default_rng(heads), torch.Generator(device="cuda").manual_seed(heads)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    tables, _, nslots = paged(rng, ctx, bs)
    if cap:
        tables = np.concatenate([tables, np.full((n, cap), -1, np.int32)], 1)
    tabs = torch.from_numpy(tables).cuda()
    cache = torch.full((nslots, row), math.nan, device="cuda", dtype=torch.bfloat16)
    rows = []
    for t in range(n):
        j = torch.arange(max(0, ctx[t] - window) if window else 0, ctx[t], device="cuda")
        rows.append(tabs[t].long()[j // bs] * bs + j % bs)
        cache[rows[t]] = 0.0
        cache[rows[t], :RANK + rot] = randn(len(j), RANK + rot).to(torch.bfloat16)
    q_abs, q = randn(n, heads * RANK) * RANK ** -0.5, randn(n, heads, dim + rot).to(torch.bfloat16)
    seq, pos = torch.arange(n, dtype=torch.int32, device="cuda"), torch.tensor(ctx, device="cuda") - 1
    out = attend(q_abs, q, seq, pos, tabs, bs, cache, heads, dim, rot, scale, window)
    for t in range(n):
        kv = cache[rows[t]].double()[:, :RANK + rot]
        x = torch.cat([q_abs[t].to(torch.bfloat16).double().reshape(heads, RANK), q[t, :, dim:].double()], -1)
        ref = torch.softmax(x @ kv.T * scale, -1) @ kv[:, :RANK]
        err = out[t].double().reshape(heads, RANK) - ref
        assert float(err.norm() / ref.norm()) < 6e-3, (t, ctx[t])


@pytest.mark.gpu
def test_a_cached_value_that_is_no_number_shows_in_its_sequence_alone(cuda):
    heads, rot, bs, dim = 16, 64, 64, 8
    ctx = [700, 900, 40]
    gen = torch.Generator(device="cuda").manual_seed(1)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    tables, _, nslots = paged(np.random.default_rng(1), ctx, bs)
    tabs = torch.from_numpy(tables).cuda()
    cache = randn(nslots, RANK + rot).to(torch.bfloat16)
    cache[int(tables[1, 3]) * bs + 5, 17] = math.nan
    q_abs, q = randn(3, heads * RANK) * 0.05, randn(3, heads * (dim + rot)).to(torch.bfloat16)
    out = attend(q_abs, q, torch.arange(3, dtype=torch.int32, device="cuda"), torch.tensor(ctx, device="cuda") - 1, tabs, bs, cache, heads, dim, rot, 0.1)
    assert out[1].isnan().all() and out[0].isfinite().all() and out[2].isfinite().all()
