"""-m gpu tests of the prompt kernel as the registered models' attentions use it (window, cap, temperature, sinks, gates; paged and dense
keys) against torch in f32, and beside the mma.sync kernel that it takes prompts from."""
import numpy as np
import pytest
import torch

from tests.util import assert_close, to_np_f32

pytestmark = pytest.mark.gpu
D = 128
# P is rounded to bf16 before P.V and the result after it: 2^-9 of a sum of weights of one, and of the result
ATOL, RTOL = 1e-2, 1.6e-2

CASES = [  # heads, kv heads, new tokens, first positions, block size (0: dense), window, cap, temperature, sinks, gate (0 none, 1 per head, 2 per value)
    (16, 4, [300, 1, 700], None, 0, 0, 0.0, 0.0, False, 0),
    (16, 4, [1024, 77, 130], None, 0, 512, 0.0, 0.0, True, 1),
    (8, 8, [257, 64], None, 0, 100, 0.0, 0.0, True, 2),
    (16, 4, [515, 200], None, 256, 0, 5.0, 0.1, False, 2),
    (6, 2, [333, 1, 128, 90], [100, 5, 64, 0], 64, 70, 0.0, 0.3, False, 1),
    (4, 1, [200, 100], [300, 63], 16, 0, 2.0, 0.0, True, 0),
    (2, 1, [100] * 40, list(range(0, 400, 10)), 128, 64, 0.0, 0.0, False, 2),
]


def _inputs(cuda, heads, kv_heads, lens, starts, bs, cap, temp, sinks, gate):
    g = torch.Generator(device="cuda").manual_seed(heads + sum(lens))
    rand = lambda *s: torch.randn(*s, generator=g, device=cuda)
    starts = starts or [0] * len(lens)
    tot = [a + n for a, n in zip(starts, lens)]
    n = sum(lens)
    ks, vs = [[rand(t, kv_heads, D).to(torch.bfloat16) for t in tot] for _ in range(2)]
    q = (2 * rand(n, heads * D)).to(torch.bfloat16)
    if bs:
        per = [-(-t // bs) for t in tot]
        ids = iter(torch.randperm(sum(per), generator=torch.Generator().manual_seed(1)).tolist())
        tables = torch.full((len(lens), max(per)), -1, dtype=torch.int32)
        kc, vc = (torch.zeros(sum(per) * bs, kv_heads * D, dtype=torch.bfloat16, device=cuda) for _ in range(2))
        for s, t in enumerate(tot):
            for b in range(per[s]):
                tables[s, b] = blk = next(ids)
                m = min(bs, t - b * bs)
                kc[blk * bs:blk * bs + m] = ks[s][b * bs:b * bs + m].flatten(1)
                vc[blk * bs:blk * bs + m] = vs[s][b * bs:b * bs + m].flatten(1)
        tables = tables.to(cuda)
    else:
        kc, vc, tables = torch.cat(ks).flatten(1), torch.cat(vs).flatten(1), None
    meta = dict(tok_seq=torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).to(torch.int32).to(cuda),
                positions=torch.cat([torch.arange(a, a + m) for a, m in zip(starts, lens)]).to(cuda),
                cu=torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device=cuda))
    gates = None if gate == 0 else rand(n, heads if gate == 1 else heads * D)
    return q, ks, vs, kc, vc, tables, meta, gates, (2 * rand(heads) if sinks else None), starts


@pytest.mark.parametrize("case", CASES, ids=[str(i) for i in range(len(CASES))])
def test_prompt_attention_against_torch(cuda, case, monkeypatch):
    from nano_vllm_rs_b200 import ops
    heads, kv_heads, lens, starts, bs, window, cap, temp, sinks, gate = case
    q, ks, vs, kc, vc, tables, meta, gates, sink, starts = _inputs(cuda, heads, kv_heads, lens, starts, bs, cap, temp, sinks, gate)
    scale, every = D ** -0.5, 50

    def call():
        return ops.window_attention(q, gates, kc, vc, meta["tok_seq"], meta["positions"], tables, bs or 256, heads, kv_heads, D, D, scale, window=window,
                                    softcap=cap, temp_coef=temp, temp_every=every, sinks=sink, gate_per_head=gate == 1, cu_tokens=meta["cu"])

    out = call()
    monkeypatch.setenv("NVLLM_CAPPED_MMA", "2")
    other = call()
    torch.cuda.synchronize()
    at = 0
    for s, n in enumerate(lens):
        pos = torch.arange(starts[s], starts[s] + n, device=cuda)
        f = scale * (1.0 + temp * torch.log(torch.floor((pos + 1) / every) + 1.0))
        rep = heads // kv_heads
        x = torch.einsum("qhd,khd->hqk", q[at:at + n].float().view(n, heads, D), ks[s].float().repeat_interleave(rep, 1)) * f[None, :, None]
        if cap:
            x = cap * torch.tanh(x / cap)
        j = torch.arange(len(ks[s]), device=cuda)
        hidden = j[None] > pos[:, None]
        if window:
            hidden = hidden | (j[None] <= pos[:, None] - window)
        x = x.masked_fill(hidden, -float("inf"))
        if sink is not None:
            x = torch.cat([x, sink[:, None, None].expand(heads, n, 1)], -1)
        p = x.softmax(-1)[..., :len(ks[s])]
        ref = torch.einsum("hqk,khd->qhd", p, vs[s].float().repeat_interleave(rep, 1))
        if gate:
            ref = ref * torch.sigmoid(gates[at:at + n].view(n, heads, -1))
        ref = to_np_f32(ref.flatten(1))
        assert_close(to_np_f32(out[at:at + n]), ref, ATOL, RTOL, f"sequence {s}")
        assert_close(to_np_f32(other[at:at + n]), ref, ATOL, RTOL, f"sequence {s} on mma.sync")
        at += n


def _causal(q, k, v, starts, window):
    """Plain causal (and windowed) attention of one sequence in f32: q [n, heads, D], k / v [keys, kv heads, D]; what a row does not see never touches it."""
    n, heads = q.shape[:2]
    pos, j = torch.arange(starts, starts + n, device=q.device), torch.arange(len(k), device=q.device)
    hidden = j[None] > pos[:, None]
    if window:
        hidden = hidden | (j[None] <= pos[:, None] - window)
    rep = heads // k.shape[1]
    x = (torch.einsum("qhd,khd->hqk", q.float(), k.float().repeat_interleave(rep, 1)) * D ** -0.5).masked_fill(hidden, -float("inf"))
    return torch.einsum("hqk,khd->qhd", x.softmax(-1), v.float().repeat_interleave(rep, 1)), ~hidden


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("heads,kv_heads,lens,starts,bs,window,sinks,gate", [
    (4, 2, [300, 77, 200], None, 0, 0, False, 0), (3, 3, [257, 130], None, 0, 100, True, 2), (8, 2, [130, 100, 333], None, 256, 0, True, 1),
    (4, 1, [200, 100], [300, 63], 16, 70, False, 2), (2, 1, [128, 128], [0, 0], 64, 0, False, 0)])
def test_no_number_reaches_only_the_tokens_that_see_it(cuda, heads, kv_heads, lens, starts, bs, window, sinks, gate, bad):
    """NaN or infinity in the values (and NaN in the keys) of every sequence's first token but the first sequence's, of one token in the middle of the
    first sequence, and in whatever its blocks hold behind its last token: a row that sees none of them is what it is without them, one that sees
    a value is not finite in that column and the same elsewhere."""
    from nano_vllm_rs_b200 import ops
    q, ks, vs, kc, vc, tables, meta, gates, sink, starts = _inputs(cuda, heads, kv_heads, lens, starts, bs, 0.0, 0.0, sinks, gate)

    def call():
        return ops.window_attention(q, gates, kc, vc, meta["tok_seq"], meta["positions"], tables, bs or 256, heads, kv_heads, D, D, D ** -0.5, window=window,
                                    sinks=sink, gate_per_head=gate == 1, cu_tokens=meta["cu"])

    clean = call()
    cu, mid, col = meta["cu"].tolist(), starts[0] + lens[0] // 2 + 3, 21
    row = lambda s, j: int(tables[s, j // bs]) * bs + j % bs if bs else cu[s] + j
    for s in range(1, len(lens)):
        kc[row(s, 0)], vc[row(s, 0)] = float("nan"), bad
    vc[row(0, mid), col] = bad                                   # one column of the first kv head
    if bs:
        for s, n in enumerate(lens):
            for j in range(starts[s] + n, -(-(starts[s] + n) // bs) * bs):
                kc[row(s, j)], vc[row(s, j)] = float("nan"), bad
    out = call()
    torch.cuda.synchronize()
    ref, seen = _causal(q[:lens[0]].view(lens[0], heads, D), ks[0], vs[0], starts[0], window)
    got, was = out[:lens[0]].view(lens[0], heads, D), clean[:lens[0]].view(lens[0], heads, D)
    hit = torch.zeros_like(got, dtype=torch.bool)
    hit[seen[:, mid], :heads // kv_heads, col] = True
    assert hit.any() and not hit.all(0).any()
    assert not torch.isfinite(got[hit]).any() and torch.isfinite(got[~hit]).all()
    assert_close(to_np_f32(got[~hit]), to_np_f32(was[~hit]), ATOL, RTOL, "rows that do not see it")
    if not sinks and not gate:
        assert_close(to_np_f32(got[~hit]), to_np_f32(ref[~hit]), ATOL, RTOL, "against torch")
    for s in range(1, len(lens)):                               # the others: rows whose window has left their first token behind
        pos = torch.arange(starts[s], starts[s] + lens[s], device=cuda)
        free = (pos >= window) if window else torch.zeros_like(pos, dtype=torch.bool)
        a, b = out[cu[s]:cu[s + 1]], clean[cu[s]:cu[s + 1]]
        assert torch.isnan(a[~free].float()).all()
        assert torch.equal(torch.isfinite(a).all(1), free)
        assert_close(to_np_f32(a[free]), to_np_f32(b[free]), ATOL, RTOL, f"sequence {s}")


def test_more_blocks_than_a_grid_has_rows(cuda):
    """7.9 million tokens in 4000 sequences: more blocks of 128 rows than the 65535 of gridDim.y."""
    from nano_vllm_rs_b200 import ops
    heads, n_seqs, L, window = 2, 4000, 1970, 64
    n = n_seqs * L
    assert n // 128 + n_seqs > 65535
    g = torch.Generator(device="cuda").manual_seed(0)
    q, k, v = (torch.randn(n, w * D, generator=g, device=cuda, dtype=torch.bfloat16) for w in (heads, 1, 1))
    cu = torch.arange(0, n + 1, L, dtype=torch.int32, device=cuda)
    out = ops.window_attention(q, None, k, v, torch.arange(n_seqs, dtype=torch.int32, device=cuda).repeat_interleave(L), torch.arange(L, device=cuda).repeat(n_seqs),
                               None, 256, heads, 1, D, D, D ** -0.5, window=window, cu_tokens=cu)
    torch.cuda.synchronize()
    for s in (0, 1999, 3999):
        rows = slice(s * L, (s + 1) * L)
        ref, _ = _causal(q[rows].view(L, heads, D), k[rows].view(L, 1, D), v[rows].view(L, 1, D), 0, window)
        assert_close(to_np_f32(out[rows]), to_np_f32(ref.flatten(1)), ATOL, RTOL, f"sequence {s}")
