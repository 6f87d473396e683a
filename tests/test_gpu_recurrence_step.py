"""Recurrences over steps of single tokens (recurrence_step.cu) against the recurrence in 64 bits and against the kernel for any step, which
the entries that do not say how many tokens there are still take."""
import pytest
import torch

DK = 128


def inputs(n, heads, groups, dv, lens, slots, pos, seed, pad):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    wide = lambda x: torch.cat([x, r(x.shape[0], pad)], 1)[:, :x.shape[1]]     # rows further apart than they are long
    k = torch.nn.functional.normalize(r(n, groups, DK), dim=-1).reshape(n, -1)
    cu = torch.tensor([0] + lens, device="cuda").cumsum(0).to(torch.int32)
    return dict(q=wide(r(n, groups * DK) * 0.3), k=wide(k), v=wide(r(n, heads * dv)), state=r(max(slots) + 1, heads, DK, dv) * 0.3,
                slots=torch.tensor(slots, device="cuda", dtype=torch.int32), cu=cu, pos=torch.tensor(pos, device="cuda"), r=r,
                u=lambda *s: torch.rand(*s, generator=gen, device="cuda"))


def in_64_bits(x, heads, groups, dv, lens, slots, pos, decay, step, skip, delta):
    """decay: [n, heads, DK or 1]; step (beta): [n, heads]."""
    state, y, t = x["state"].double().clone(), torch.zeros(x["v"].shape[0], heads, dv, dtype=torch.float64, device="cuda"), 0
    d = heads // groups
    for s, ln in enumerate(lens):
        S = state[slots[s]].clone() if slots[s] >= 0 else None
        for i in range(ln):
            if S is not None:
                if i == 0 and pos[t] == 0:
                    S.zero_()
                k, q = (x[c][t].double().reshape(groups, DK).repeat_interleave(d, 0) for c in "kq")
                v, b = x["v"][t].double().reshape(heads, dv), step[t].double()[:, None]
                S = S * decay[t].double()[..., None]
                u = b * (v - torch.einsum("hkv,hk->hv", S, k)) if delta else b * v
                S = S + k[..., None] * u[:, None]
                y[t] = torch.einsum("hkv,hk->hv", S, q) + (skip.double()[:, None] * v if skip is not None else 0.0)
            t += 1
        if S is not None and ln:
            state[slots[s]] = S
    return y.reshape(y.shape[0], -1), state


CASES = [   # heads, groups, dv, tokens of each sequence (as many as sequences), slots, position of each sequence's first token
    (4, 2, 64, [1, 1, 1], [2, 0, 1], [7, 0, 3]),                 # one starts anew
    (3, 3, 96, [1, 1], [1, -1], [4, 4]),                         # a padding row of a graph; columns that only 32 divides
    (16, 4, 128, [1] * 40, list(range(39, -1, -1)), [9] * 40),   # slices of 128 columns
    (6, 2, 256, [2, 0, 1, 1], [0, 3, 1, 2], [0, 5, 1, 8]),       # as many tokens as sequences, but not one each
    (16, 1, 64, [1] * 33, list(range(33)), [5] * 33)]


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.gpu
@pytest.mark.parametrize("heads,groups,dv,lens,slots,pos", CASES)
@pytest.mark.parametrize("full", [True, False])
def test_linear_recurrence_of_single_tokens(cuda, heads, groups, dv, lens, slots, pos, full):
    """The state is, to the bit, what the other kernel keeps; the read-out sums 128 products in another order (2^-24 each, a few of them
    rounding the same way: 1e-6 of the result)."""
    from nano_vllm_rs_b200 import _ffi
    n = sum(lens)
    at = [p for p, ln in zip(pos, lens) for p in range(p, p + ln)]
    x = inputs(n, heads, groups, dv, lens, slots, at, heads + dv, 3)
    decay = 0.8 + 0.2 * x["u"](n, heads) if full else 0.8 + 0.2 * x["u"](heads)
    step, skip = (x["u"](n, heads), x["r"](heads)) if full else (None, None)
    ref, S = in_64_bits(x, heads, groups, dv, lens, slots, at, (decay if full else decay.expand(n, heads))[..., None], step if full else torch.ones(n, heads, device="cuda"), skip, False)
    p = lambda t: t.data_ptr() if t is not None else None
    got = []
    for entry, tokens in (("nvllm_linear_recurrence_step", [n]), ("nvllm_linear_recurrence", [])):
        state, y = x["state"].clone(), torch.full((n, heads * dv), 7.0, device="cuda")
        _ffi.check(getattr(_ffi.lib(), entry)(p(y), y.stride(0), p(x["q"]), x["q"].stride(0), p(x["k"]), x["k"].stride(0), p(x["v"]), x["v"].stride(0), p(decay), int(full), p(step), int(full),
                                              p(skip), p(state), p(x["slots"]), p(x["cu"]), p(x["pos"]), *tokens, len(lens), heads, groups, DK, dv, torch.cuda.current_stream().cuda_stream))
        got.append((y, state))
    (y, state), (y0, state0) = got
    assert torch.equal(state, state0) and rel(state, S) < 3e-7
    assert rel(y, ref) < 1e-6 and rel(y, ref) < 1.2 * rel(y0, ref) + 2e-8


@pytest.mark.gpu
@pytest.mark.parametrize("heads,groups,dv,lens,slots,pos", CASES)
@pytest.mark.parametrize("channel", [True, False])
def test_delta_rule_of_single_tokens(cuda, heads, groups, dv, lens, slots, pos, channel):
    """As above; u carries a sum of 128 products into the state as well."""
    from nano_vllm_rs_b200 import _ffi
    n = sum(lens)
    at = [p for p, ln in zip(pos, lens) for p in range(p, p + ln)]
    x = inputs(n, heads, groups, dv, lens, slots, at, heads + dv, 5)
    decay, beta = 0.8 + 0.2 * x["u"](n, heads * (DK if channel else 1)), x["u"](n, heads)
    ref, S = in_64_bits(x, heads, groups, dv, lens, slots, at, decay.reshape(n, heads, -1), beta, None, True)
    p = lambda t: t.data_ptr()
    got = []
    for tokens in (n, 0):
        state, y = x["state"].clone(), torch.full((n, heads * dv), 7.0, device="cuda")
        _ffi.check(_ffi.lib().nvllm_delta_recurrence_step(p(y), y.stride(0), p(x["q"]), x["q"].stride(0), p(x["k"]), x["k"].stride(0), p(x["v"]), x["v"].stride(0), p(decay), decay.stride(0),
                                                          int(not channel), p(beta), heads, p(state), p(x["slots"]), p(x["cu"]), p(x["pos"]), tokens, len(lens), heads, groups, DK, dv,
                                                          torch.cuda.current_stream().cuda_stream))
        got.append((y, state))
    (y, state), (y0, state0) = got
    assert rel(state, S) < 3e-7 and rel(state, S) < 1.1 * rel(state0, S) + 1e-8
    assert rel(y, ref) < 1e-6 and rel(y, ref) < 1.2 * rel(y0, ref) + 2e-8
