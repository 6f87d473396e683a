"""Latent attention of prompts and portions on tcgen05 (kv_rank 512), the split of single tokens' keys, and what falls to the
mma.sync kernel beside them, against the attention in 64 bits."""
import math

import numpy as np
import pytest
import torch

from tests.arch_util import paged

RANK = 512


def reference(q_abs, q_rot, cache, spans, pos, tables, bs, heads, rot, scale, window, sinks, gate):
    out = torch.empty(q_abs.shape[0], heads, RANK, dtype=torch.float64, device=q_abs.device)
    for s, (a, b) in enumerate(spans):
        L = int(pos[a:b].max()) + 1
        j = torch.arange(L, device=q_abs.device)
        rows = cache[(tables[s].long()[j // bs] * bs + j % bs)].double()
        x = torch.cat([q_abs[a:b].to(torch.bfloat16).double().reshape(b - a, heads, RANK), q_rot[a:b].double()], -1)
        sc = x @ rows[:, :RANK + rot].T * scale
        hidden = j[None] > pos[a:b, None]
        if window:
            hidden |= j[None] <= pos[a:b, None] - window
        sc = sc.masked_fill(hidden[:, None], -math.inf)
        if sinks is not None:
            sc = torch.cat([sc, sinks.double()[None, :, None].expand(b - a, heads, 1)], -1)
        p = torch.softmax(sc, -1)[..., :L]
        o = p @ rows[:, :RANK]
        out[a:b] = o if gate is None else o * torch.sigmoid(gate[a:b].double())[..., None]
    return out.reshape(q_abs.shape[0], -1)


@pytest.mark.gpu
@pytest.mark.parametrize("heads,rot,bs,window,extras,portions", [
    (16, 64, 16, 0, False, [(0, 64), (0, 1), (130, 9), (3, 70)]),      # prompts, a single token, portions behind cached keys
    (16, 64, 256, 0, False, [(0, 8), (0, 8), (0, 8), (0, 8)]),         # every tile one sequence
    (32, 8, 48, 100, True, [(0, 63), (500, 65), (63, 1), (64, 2)]),    # two head groups, a window, sinks and a gate
    (16, 0, 16, 33, True, [(0, 129), (0, 127)]),                       # no rotated part
    (16, 64, 64, 0, False, [(k * 17, 1) for k in range(40)]),          # single tokens alone: no dense tile
    (16, 64, 64, 0, False, [(40, 1), (0, 100), (700, 1), (5, 1), (9, 1), (2, 1), (1000, 30)]),
    (16, 64, 256, 0, False, [(1500, 1), (700, 1), (0, 1)]),            # few single tokens: their keys are split over CTAs
])
def test_latent_prompts_portions_and_single_tokens(cuda, heads, rot, bs, window, extras, portions):
    from nano_vllm_rs_b200 import _ffi, ops
    rng = np.random.default_rng(len(portions) + heads + rot)
    gen = torch.Generator(device="cuda").manual_seed(7)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    dim, row = 24, RANK + rot
    ctx = [c + n for c, n in portions]
    tables, _, nslots = paged(rng, ctx, bs)
    cache = randn(nslots, row).to(torch.bfloat16)
    counts = [n for _, n in portions]
    N = sum(counts)
    starts = np.concatenate([[0], np.cumsum(counts)])
    spans = [(int(starts[i]), int(starts[i + 1])) for i in range(len(counts))]
    pos = torch.cat([torch.arange(c, c + n) for c, n in portions]).cuda()
    tok_seq = torch.repeat_interleave(torch.arange(len(counts)), torch.tensor(counts)).to(torch.int32).cuda()
    tabs = torch.from_numpy(tables).cuda()
    q_abs = randn(N, heads * RANK) * 0.5
    q = randn(N, heads, dim + rot).to(torch.bfloat16)
    scale = 0.11
    sinks = randn(heads) if extras else None
    gate = randn(N, heads) if extras else None
    if extras:
        got = out = torch.empty((N, heads * RANK), dtype=torch.bfloat16, device="cuda")
        p = lambda t: t.data_ptr()
        _ffi.check(_ffi.lib().nvllm_latent_window_attention(p(out), out.stride(0), p(q_abs), q_abs.stride(0), p(q), q.stride(0), p(tok_seq), p(pos), p(tabs),
                                                            tabs.shape[1], bs, p(cache), cache.stride(0), N, heads, dim, rot, RANK, scale, window,
                                                            p(sinks), p(gate), heads, None, 0, 0, torch.cuda.current_stream().cuda_stream))
    else:
        got = ops.latent_attention(q_abs, q.reshape(N, -1), tok_seq, pos, tabs, bs, cache, heads, dim, rot, RANK, scale)
    ref = reference(q_abs, q[..., dim:], cache, spans, pos, tabs, bs, heads, rot, scale, window, sinks, gate)
    # bf16 probabilities (2^-9 each) against exact ones, and a bf16 output (2^-9): per value of O(1)
    err = (got.double() - ref).abs()
    assert torch.isfinite(got.float()).all()
    assert float((err / (ref.abs() + 0.25 * ref.pow(2).mean().sqrt())).max()) < 0.06, float(err.max())
    assert float(err.norm() / ref.norm()) < 6e-3


def call(q_abs, q, tok_seq, pos, tabs, bs, cache, heads, dim, rot, scale, window=0):
    """The C entry without a workspace: nothing is split."""
    from nano_vllm_rs_b200 import _ffi
    out = torch.empty((q.shape[0], heads * RANK), dtype=torch.bfloat16, device="cuda")
    p = lambda t: t.data_ptr()
    _ffi.check(_ffi.lib().nvllm_latent_window_attention(p(out), out.stride(0), p(q_abs), q_abs.stride(0), p(q), q.stride(0), p(tok_seq), p(pos), p(tabs), tabs.shape[1],
                                                        bs, p(cache), cache.stride(0), q.shape[0], heads, dim, rot, RANK, scale, window, None, None, 0, None, 0, 0,
                                                        torch.cuda.current_stream().cuda_stream))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("n", [32, 33, 34, 40, 41, 42])
def test_single_tokens_are_what_each_gives_alone(cuda, n):
    """Single tokens keep to the kernel of single tokens whatever their number is (a last tile of one or two is no prompt): without a
    split every row is, to the bit, what its token gives alone."""
    heads, dim, rot, bs, scale = 16, 24, 64, 64, 0.11
    rng = np.random.default_rng(n)
    gen = torch.Generator(device="cuda").manual_seed(n)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    ctx = rng.integers(1, 700, n)
    ctx[-2:] = 650, 333
    tables, _, nslots = paged(rng, [int(c) for c in ctx], bs)
    cache, tabs = randn(nslots, RANK + rot).to(torch.bfloat16), torch.from_numpy(tables).cuda()
    q_abs, q = randn(n, heads * RANK) * 0.5, randn(n, heads * (dim + rot)).to(torch.bfloat16)
    seq, pos = torch.arange(n, dtype=torch.int32, device="cuda"), torch.from_numpy(ctx - 1).cuda()
    got = call(q_abs, q, seq, pos, tabs, bs, cache, heads, dim, rot, scale)
    for t in range(n):
        alone = call(q_abs[t:t + 1], q[t:t + 1], seq[t:t + 1], pos[t:t + 1], tabs, bs, cache, heads, dim, rot, scale)
        assert torch.equal(alone[0], got[t]), t


@pytest.mark.gpu
@pytest.mark.parametrize("value", [math.nan, math.inf, -math.inf])
@pytest.mark.parametrize("column", [3, 300, RANK + 5])   # either half of the latent values, the rotated part
@pytest.mark.parametrize("window,tokens", [(0, 129), (33, 129), (0, 1200)])   # 1200: both halves in one CTA
def test_a_cached_value_that_is_no_number_stays_with_the_tokens_that_see_it(cuda, value, column, window, tokens):
    """Tokens of a tile share the key tiles; a key that a token does not see must not reach it through 0 x Inf."""
    heads, dim, rot, bs, scale, at = 16, 24, 64, 64, 0.11, 50
    gen = torch.Generator(device="cuda").manual_seed(tokens + column)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    tables, _, nslots = paged(np.random.default_rng(1), [tokens], bs)
    cache, tabs = randn(nslots, RANK + rot).to(torch.bfloat16), torch.from_numpy(tables).cuda()
    q_abs, q = randn(tokens, heads * RANK) * 0.5, randn(tokens, heads, dim + rot).to(torch.bfloat16)
    seq, pos = torch.zeros(tokens, dtype=torch.int32, device="cuda"), torch.arange(tokens, device="cuda")
    ref = reference(q_abs, q[..., dim:], cache, [(0, tokens)], pos, tabs, bs, heads, rot, scale, window, None, None)
    cache[int(tables[0, at // bs]) * bs + at % bs, column] = value
    got = call(q_abs, q.reshape(tokens, -1), seq, pos, tabs, bs, cache, heads, dim, rot, scale, window).double()
    sees = (pos >= at) & ((pos < at + window) if window else True)
    err = (got - ref)[~sees]
    assert torch.isfinite(got[~sees]).all()
    assert float(err.norm() / ref[~sees].norm()) < 6e-3 and float((err.abs() / (ref[~sees].abs() + 0.25 * ref.pow(2).mean().sqrt())).max()) < 0.06
    if value != value:
        assert not torch.isfinite(got[sees]).any()


def kernels_of(f):
    """How many kernels f launches: the nodes of its graph."""
    from cuda.bindings import runtime
    f()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        f()
    err, _, count = runtime.cudaGraphGetNodes(runtime.cudaGraph_t(graph.raw_cuda_graph()))
    assert int(err) == 0
    return int(count)


@pytest.mark.gpu
@pytest.mark.parametrize("n,context,launches", [(8, 300, 1), (40, 300, 1), (40, 3000, 2), (300, 300, 1)])
def test_a_batch_of_single_tokens_launches_no_kernel_for_prompts(cuda, n, context, launches):
    from nano_vllm_rs_b200 import ops
    heads, dim, rot, bs, scale = 16, 24, 64, 64, 0.11
    gen = torch.Generator(device="cuda").manual_seed(n)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    tables, _, nslots = paged(np.random.default_rng(n), [context] * n, bs)
    cache, tabs = randn(nslots, RANK + rot).to(torch.bfloat16), torch.from_numpy(tables).cuda()
    q_abs, q = randn(n, heads * RANK) * 0.5, randn(n, heads * (dim + rot)).to(torch.bfloat16)
    seq, pos = torch.arange(n, dtype=torch.int32, device="cuda"), torch.full((n,), context - 1, device="cuda")
    run = lambda: ops.latent_attention(q_abs, q, seq, pos, tabs, bs, cache, heads, dim, rot, RANK, scale)
    assert kernels_of(run) == launches
    if launches == 1:
        assert torch.equal(run(), call(q_abs, q, seq, pos, tabs, bs, cache, heads, dim, rot, scale))


@pytest.mark.gpu
def test_the_entry_of_single_tokens_takes_any_batch(cuda, monkeypatch):
    """Prompts and portions given to nvllm_latent_token_attention run on the mma.sync kernel."""
    from nano_vllm_rs_b200 import _ffi
    heads, dim, rot, bs, scale = 16, 24, 64, 64, 0.11
    gen = torch.Generator(device="cuda").manual_seed(3)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    counts = [70, 1, 30]
    n = sum(counts)
    tables, _, nslots = paged(np.random.default_rng(3), counts, bs)
    cache, tabs = randn(nslots, RANK + rot).to(torch.bfloat16), torch.from_numpy(tables).cuda()
    q_abs, q = randn(n, heads * RANK) * 0.5, randn(n, heads * (dim + rot)).to(torch.bfloat16)
    seq = torch.repeat_interleave(torch.arange(3), torch.tensor(counts)).to(torch.int32).cuda()
    pos = torch.cat([torch.arange(c) for c in counts]).cuda()
    args = (q_abs, q, seq, pos, tabs, bs, cache, heads, dim, rot, scale)
    prompts = call(*args)
    with monkeypatch.context() as m:
        m.setattr(_ffi.lib(), "nvllm_latent_window_attention", _ffi.lib().nvllm_latent_token_attention)
        single = call(*args)
    monkeypatch.setenv("NVLLM_LATENT_MMA", "2")
    assert torch.equal(single, call(*args)) and not torch.equal(single, prompts)


@pytest.mark.gpu
def test_a_workspace_is_asked_for_where_keys_can_be_split(cuda, monkeypatch):
    """Eight tiles of 64 keys are the fewest that two CTAs share; the split never lies below."""
    from nano_vllm_rs_b200 import _ffi, ops
    heads, dim, rot, scale, n = 16, 24, 64, 0.11, 4
    gen = torch.Generator(device="cuda").manual_seed(5)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    asked = []
    entry = _ffi.lib().nvllm_latent_workspace_bytes
    monkeypatch.setattr(_ffi.lib(), "nvllm_latent_workspace_bytes", lambda *a: asked.append(a) or entry(*a))
    q_abs, q, seq = randn(n, heads * RANK) * 0.5, randn(n, heads * (dim + rot)).to(torch.bfloat16), torch.arange(n, dtype=torch.int32, device="cuda")
    for blocks, launches in ((7, 1), (8, 2)):
        tabs = torch.arange(n * blocks, dtype=torch.int32, device="cuda").reshape(n, blocks)
        cache, pos = randn(n * blocks * 64, RANK + rot).to(torch.bfloat16), torch.full((n,), blocks * 64 - 1, device="cuda")
        ws = torch.empty(entry(n, heads, RANK) // 4, device="cuda")
        asked.clear()
        assert kernels_of(lambda: ops.latent_attention(q_abs, q, seq, pos, tabs, 64, cache, heads, dim, rot, RANK, scale)) == launches
        assert bool(asked) == (launches == 2)
        assert kernels_of(lambda: ops.latent_rotary_attention(q_abs, q, seq, pos, tabs, 64, cache, heads, dim, rot, RANK, scale, workspace=ws)) == launches
