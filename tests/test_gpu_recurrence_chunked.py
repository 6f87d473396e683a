"""-m gpu tests of the linear recurrence's kernel for prompts (32 tokens at a time as matrix products) against the token-by-token
recurrence in float64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DK = 128
# A result is a sum of products a ... a b k v q.  The split operands keep 2^-24 of a product (three of its nine parts are left out), the
# accumulators are f32: over up to 128 keys and the chunks before, 64 roundings of 2^-24 bound what does not average out.
TOL = 67 * 2.0 ** -24


def _reference(q, k, v, a, b, d, S):
    """One sequence in float64: y [n, heads, dv], the final state, and the same with all values' magnitudes (the error's scale)."""
    n, H, dv = v.shape
    y, B, Sb = np.empty_like(v), np.empty_like(v), np.abs(S)
    S = S.copy()
    with np.errstate(all="ignore"):
        for t in range(n):
            S = a[t][:, None, None] * S + (b[t][:, None] * k[t])[:, :, None] * v[t][:, None, :]
            y[t] = np.einsum("hkv,hk->hv", S, q[t]) + d[:, None] * v[t]
            Sb = np.abs(a[t])[:, None, None] * Sb + (np.abs(b[t])[:, None] * np.abs(k[t]))[:, :, None] * np.abs(v[t])[:, None, :]
            B[t] = np.einsum("hkv,hk->hv", Sb, np.abs(q[t])) + np.abs(d)[:, None] * np.abs(v[t])
    return y, S, B, Sb


def _run(cuda, seqs, heads, groups, dv, state, starts, per_token, skip):
    """seqs: per sequence a dict of q, k [n, groups, DK], v [n, heads, dv], a, b [n, heads] (f32); state [slots, heads, DK, dv] on the device."""
    from nano_vllm_rs_b200 import ops
    cat = lambda x, w: torch.from_numpy(np.concatenate([s[x].reshape(len(s["v"]), w) for s in seqs])).to(cuda)
    lens = [len(s["v"]) for s in seqs]
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device=cuda)
    pos = torch.cat([torch.arange(p, p + n) for p, n in zip(starts, lens)]).to(cuda)
    slots = torch.arange(len(seqs), dtype=torch.int32, device=cuda)
    a, b = cat("a", heads), cat("b", heads)
    y = ops.linear_recurrence(cat("q", groups * DK), cat("k", groups * DK), cat("v", heads * dv), a if per_token else a[0].contiguous(), state, slots, cu,
                              pos, heads, groups, DK, dv, step=b if per_token else b[0].contiguous(), skip=None if skip is None else torch.from_numpy(skip).to(cuda))
    return np.split(y.cpu().numpy().reshape(-1, heads, dv), np.cumsum(lens)[:-1])


def _seq(rng, n, heads, groups, dv, per_token=True, scale=1.0):
    f = lambda x: np.asarray(x, np.float32)
    a = rng.uniform(0.6, 1.0, (n, heads)) if per_token else np.tile(1.0 - 2.0 ** -np.linspace(3, 9, heads), (n, 1))
    b = rng.uniform(0.1, 1.0, (n, heads)) if per_token else np.full((n, heads), 0.09)
    return {"q": f(rng.standard_normal((n, groups, DK))), "k": f(scale * rng.standard_normal((n, groups, DK))), "v": f(rng.standard_normal((n, heads, dv))), "a": f(a), "b": f(b)}


def _check(seq, S0, got, state, heads, groups, d):
    w = {x: s.astype(np.float64) for x, s in seq.items()}
    rep = heads // groups
    y, S, B, Sb = _reference(w["q"].repeat(rep, 1), w["k"].repeat(rep, 1), w["v"], w["a"], w["b"], d, S0)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(y))
    np.testing.assert_array_equal(np.isinf(got), np.isinf(y))
    ok = np.isfinite(y)
    assert (np.abs(got - y)[ok] <= TOL * B[ok] + 1e-30).all(), np.max(np.abs(got - y)[ok] / (B[ok] + 1e-30))
    ok = np.isfinite(S)
    np.testing.assert_array_equal(np.isfinite(state), ok)
    assert (np.abs(state - S)[ok] <= TOL * Sb[ok] + 1e-30).all()
    return S


@pytest.mark.parametrize("heads,groups,dv,lens,per_token", [
    (2, 2, 64, [16], True), (4, 2, 64, [31, 1, 64], True), (8, 1, 64, [33, 97], True), (3, 3, 128, [32, 130], False), (2, 1, 192, [65, 40], True)])
def test_prompts_and_portions(cuda, heads, groups, dv, lens, per_token):
    """Chunk edges and tails, single tokens beside prompts, a second portion that continues from the slots, a fresh one that ignores them."""
    rng = np.random.default_rng(sum(lens) + dv)
    skip = np.asarray(rng.standard_normal(heads), np.float32) if per_token else None
    d = np.zeros(heads) if skip is None else skip.astype(np.float64)
    state = torch.full((len(lens), heads, DK, dv), 7.0, device=cuda)
    S = [np.zeros((heads, DK, dv))] * len(lens)
    for portion in range(2):
        seqs = [_seq(rng, n, heads, groups, dv, per_token) for n in lens]
        ys = _run(cuda, seqs, heads, groups, dv, state, [portion * n for n in lens], per_token, skip)
        st = state.cpu().numpy()
        S = [_check(q, s, y, st[i], heads, groups, d) for i, (q, s, y) in enumerate(zip(seqs, S, ys))]
        S = [torch.from_numpy(st[i]).double().numpy() for i in range(len(lens))]   # the next portion starts from the f32 state


@pytest.mark.parametrize("what", ["v nan", "v inf", "k nan", "q inf", "a zero", "a above one", "a nan", "k large", "k tiny", "all zero"])
def test_odd_values(cuda, what):
    """What a value out of the ordinary reaches: later tokens of its sequence and head, of its column if it is v's, nothing before it."""
    heads, groups, dv, n, at = 4, 2, 64, 100, 45
    rng = np.random.default_rng(7)
    seqs = [_seq(rng, n, heads, groups, dv), _seq(rng, n, heads, groups, dv)]
    s = seqs[0]
    if what == "v nan": s["v"][at, 1, 5] = np.nan
    elif what == "v inf": s["v"][at, 1, 5] = np.inf
    elif what == "k nan": s["k"][at, 0, 3] = np.nan
    elif what == "q inf": s["q"][at, 1, 9] = np.inf
    elif what == "a zero": s["a"][at] = 0.0
    elif what == "a above one": s["a"][at:at + 3] = 1.5
    elif what == "a nan": s["a"][at, 2] = np.nan
    elif what == "k large": s["k"][at] *= np.float32(2.0 ** 50)
    elif what == "k tiny": s["k"][at] *= np.float32(2.0 ** -100)
    else:
        for x in "qkv": s[x][:] = 0.0
    state = torch.zeros((2, heads, DK, dv), device=cuda)
    ys = _run(cuda, seqs, heads, groups, dv, state, [0, 0], True, None)
    st = state.cpu().numpy()
    for i in range(2):
        _check(seqs[i], np.zeros((heads, DK, dv)), ys[i], st[i], heads, groups, np.zeros(heads))
