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
