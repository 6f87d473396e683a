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
    (32, 64, 16, 0, False, [(0, 64), (0, 1), (130, 9), (3, 70)]),      # prompts, a single token, portions behind cached keys
    (16, 64, 256, 0, False, [(0, 8)] * 40),                            # every tile one sequence
    (32, 8, 48, 100, True, [(0, 63), (500, 65), (63, 1), (64, 2)]),    # two head groups, a window, sinks and a gate
    (16, 0, 16, 33, True, [(0, 129), (0, 127)]),                       # no rotated part
    (16, 64, 64, 0, False, [(k * 17, 1) for k in range(40)]),          # single tokens alone
    (16, 64, 64, 0, True, [(k * 3, 1) for k in range(170)]),           # as many that the kernel for prompts is tried: no dense tile
    (32, 64, 64, 0, False, [(40, 1), (0, 100), (700, 1), (5, 1), (9, 1), (2, 1), (1000, 30)]),
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


def call(q_abs, q, tok_seq, pos, tabs, bs, cache, heads, dim, rot, scale, window=0, n_seqs=None):
    """The C entries that do not say how many sequences the batch holds, and that do."""
    from nano_vllm_rs_b200 import _ffi
    lib = _ffi.lib()
    out = torch.empty((q.shape[0], heads * RANK), dtype=torch.bfloat16, device="cuda")
    p = lambda t: t.data_ptr()
    head = (p(out), out.stride(0), p(q_abs), q_abs.stride(0), p(q), q.stride(0), p(tok_seq), p(pos), p(tabs), tabs.shape[1], bs, p(cache), cache.stride(0), q.shape[0])
    rest = (heads, dim, rot, RANK, scale, window, None, None, 0, None, 0, 0, torch.cuda.current_stream().cuda_stream)
    _ffi.check(lib.nvllm_latent_window_attention(*head, *rest) if n_seqs is None else lib.nvllm_latent_step_attention(*head, n_seqs, *rest))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("n", [33, 152, 153, 154, 162])
def test_single_tokens_are_what_each_gives_alone(cuda, n):
    """Single tokens keep to the kernel of single tokens whatever their number is (a last tile of one or two is no prompt): in tables of
    three tiles of keys, which no CTAs share, every row is, to the bit, what its token gives alone."""
    heads, dim, rot, bs, scale = 16, 24, 64, 64, 0.11
    rng = np.random.default_rng(n)
    gen = torch.Generator(device="cuda").manual_seed(n)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    ctx = rng.integers(1, 193, n)
    ctx[-2:] = 192, 130
    tables, _, nslots = paged(rng, [int(c) for c in ctx], bs)
    tables = tables[:, :3].copy()
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
    heads, dim, rot, bs, scale, at = 32, 24, 64, 64, 0.11, 50
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
@pytest.mark.parametrize("n,context,launches", [(1, 20, 1), (8, 300, 1), (40, 300, 1), (40, 3000, 1), (300, 300, 1)])
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
    assert torch.equal(run(), call(q_abs, q, seq, pos, tabs, bs, cache, heads, dim, rot, scale))


@pytest.mark.gpu
def test_the_number_of_sequences_only_chooses_the_kernel(cuda, monkeypatch):
    """A caller that says 'single tokens' about prompts gets them from the mma.sync kernel; the right number changes nothing."""
    heads, dim, rot, bs, scale = 32, 24, 64, 64, 0.11
    gen = torch.Generator(device="cuda").manual_seed(3)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    counts = [70, 1, 100]
    n = sum(counts)
    tables, _, nslots = paged(np.random.default_rng(3), counts, bs)
    cache, tabs = randn(nslots, RANK + rot).to(torch.bfloat16), torch.from_numpy(tables).cuda()
    q_abs, q = randn(n, heads * RANK) * 0.5, randn(n, heads * (dim + rot)).to(torch.bfloat16)
    seq = torch.repeat_interleave(torch.arange(3), torch.tensor(counts)).to(torch.int32).cuda()
    pos = torch.cat([torch.arange(c) for c in counts]).cuda()
    args = (q_abs, q, seq, pos, tabs, bs, cache, heads, dim, rot, scale)
    prompts = call(*args)
    assert torch.equal(prompts, call(*args, n_seqs=3)) and torch.equal(prompts, call(*args, n_seqs=0))
    single = call(*args, n_seqs=n)
    monkeypatch.setenv("NVLLM_LATENT_MMA", "2")
    assert torch.equal(single, call(*args)) and not torch.equal(single, prompts)


@pytest.mark.gpu
@pytest.mark.parametrize("heads,rank,rot", [(16, 512, 64), (40, 512, 0), (5, 512, 8), (16, 96, 64), (3, 30, 2), (16, 200, 16), (17, 384, 64)])
@pytest.mark.parametrize("n,extras", [(1, False), (3, True), (11, False), (37, True)])
def test_clusters_share_the_keys_of_single_tokens(cuda, heads, rank, rot, n, extras):
    """Contexts around the edges of tiles and shares, in tables that allow far longer ones: one CTA, some or all of a cluster have
    keys; sinks and gates join in the merge; an unused row of a graph has no key at all."""
    from nano_vllm_rs_b200 import _ffi
    bs, dim, scale, row = 48, 8, 0.3, -(-(rank + rot) // 8) * 8
    rng = np.random.default_rng(n + heads)
    gen = torch.Generator(device="cuda").manual_seed(n + rank)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    ctx = [int(c) for c in rng.choice([1, 63, 64, 65, 127, 128, 129, 191, 193, 255, 256, 257, 320, 700, 1025, 2000], n)]
    ctx[0] = 1501
    tables, _, nslots = paged(rng, ctx, bs)
    tables = np.concatenate([tables, np.full((n, 90), -1, np.int32)], 1)
    if n > 3:
        tables[2] = -1
    cache, tabs = torch.zeros(nslots, row, device="cuda", dtype=torch.bfloat16), torch.from_numpy(tables).cuda()
    cache[:, :rank + rot] = randn(nslots, rank + rot).to(torch.bfloat16)
    q_abs, q = randn(n, heads * rank) * rank ** -0.5, randn(n, heads, dim + rot).to(torch.bfloat16)
    seq, pos = torch.arange(n, dtype=torch.int32, device="cuda"), torch.tensor(ctx, device="cuda") - 1
    sinks, gate = (randn(heads), randn(n, heads)) if extras else (None, None)
    out = torch.full((n, heads * rank), 7.0, dtype=torch.bfloat16, device="cuda")
    p = lambda t: t.data_ptr() if t is not None else None
    _ffi.check(_ffi.lib().nvllm_latent_step_attention(p(out), out.stride(0), p(q_abs), q_abs.stride(0), p(q), q.stride(0), p(seq), p(pos), p(tabs), tabs.shape[1],
                                                      bs, p(cache), row, n, n, heads, dim, rot, rank, scale, 0, p(sinks), p(gate), heads, None, 0, 0,
                                                      torch.cuda.current_stream().cuda_stream))
    for t in range(n):
        if n > 3 and t == 2:
            assert (out[t] == 0).all()
            continue
        j = torch.arange(ctx[t], device="cuda")
        rows = cache[tabs[t].long()[j // bs] * bs + j % bs].double()
        x = torch.cat([q_abs[t].to(torch.bfloat16).double().reshape(heads, rank), q[t, :, dim:].double()], -1)
        sc = x @ rows[:, :rank + rot].T * scale
        if extras:
            sc = torch.cat([sc, sinks.double()[:, None]], 1)
        ref = torch.softmax(sc, -1)[:, :ctx[t]] @ rows[:, :rank]
        if extras:
            ref = ref * torch.sigmoid(gate[t].double())[:, None]
        err = out[t].double().reshape(heads, rank) - ref
        assert float(err.norm() / ref.norm()) < 6e-3, (t, ctx[t])


@pytest.mark.gpu
@pytest.mark.parametrize("heads,window,extras", [(48, 0, False), (64, 50, True)])
def test_what_is_left_of_prompts_with_many_heads(cuda, heads, window, extras):
    """Up to 256 tokens whose few tiles of many sequences go to the mma.sync kernel behind the prompts: more than two CTAs an SM would have nothing to do elsewhere."""
    test_latent_prompts_portions_and_single_tokens(cuda, heads, 64, 64, window, extras, [(40, 1), (0, 100), (700, 1), (5, 1), (9, 1), (2, 1), (1000, 30)])
