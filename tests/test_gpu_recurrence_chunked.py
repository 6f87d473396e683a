"""-m gpu tests of the recurrences' kernels for prompts (32 or 16 tokens at a time as matrix products) against the token-by-token
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


# ------------------------------------------------------------------------------------------------------------ the gated delta rule
def _delta_reference(q, k, v, g, b, S):
    """One sequence in float64: y, the final state, and the largest column norm that the state had (the error's scale)."""
    n, H, dv = v.shape
    y, S, top = np.empty_like(v), S.copy(), np.zeros((H, dv))
    with np.errstate(all="ignore"):
        for t in range(n):
            S = g[t][:, :, None] * S
            u = b[t][:, None] * (v[t] - np.einsum("hkv,hk->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            y[t] = np.einsum("hkv,hk->hv", S, q[t])
            top = np.fmax(top, np.sqrt((S * S).sum(1)))
    return y, S, top


def _delta_seq(rng, n, heads, groups, dv, head_decay, lo=0.5):
    f = lambda x: np.asarray(x, np.float32)
    unit = lambda x: x / np.sqrt((x * x).sum(-1, keepdims=True))
    return {"q": f(unit(rng.standard_normal((n, groups, DK)))), "k": f(unit(rng.standard_normal((n, groups, DK)))), "v": f(rng.standard_normal((n, heads, dv))),
            "g": f(rng.uniform(lo, 1.0, (n, heads, 1 if head_decay else DK))), "b": f(rng.uniform(0.1, 1.0, (n, heads)))}


def _delta_run(cuda, seqs, heads, groups, dv, state, starts, head_decay):
    from nano_vllm_rs_b200 import ops
    cat = lambda x: torch.from_numpy(np.concatenate([s[x].reshape(len(s["v"]), -1) for s in seqs])).to(cuda)
    lens = [len(s["v"]) for s in seqs]
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device=cuda)
    pos = torch.cat([torch.arange(p, p + n) for p, n in zip(starts, lens)]).to(cuda)
    slots = torch.arange(len(seqs), dtype=torch.int32, device=cuda)
    fn = ops.head_delta_recurrence if head_decay else ops.gated_delta_recurrence
    y = fn(cat("q"), cat("k"), cat("v"), cat("g"), cat("b"), state, slots, cu, pos, heads, groups, DK, dv)
    return np.split(y.cpu().numpy().reshape(-1, heads, dv), np.cumsum(lens)[:-1])


def _delta_check(seq, S0, got, state, heads, groups, tokens):
    """With unit keys and beta <= 1 a step never enlarges an error that the state carries, so the errors of the tokens so far add up at the
    worst; each is a handful (16 are allowed) of roundings of 2^-24 on the scale of a state's column."""
    w = {x: s.astype(np.float64) for x, s in seq.items()}
    rep = heads // groups
    y, S, top = _delta_reference(w["q"].repeat(rep, 1), w["k"].repeat(rep, 1), w["v"], np.broadcast_to(w["g"], w["g"].shape[:2] + (DK,)), w["b"], S0)
    tol = tokens * 16 * 2.0 ** -24 * np.where(np.isfinite(top), np.maximum(top, 1e-30), 1.0)
    np.testing.assert_array_equal(np.isfinite(got), np.isfinite(y))
    ok = np.isfinite(y)
    with np.errstate(invalid="ignore"):
        assert (np.abs(got - y)[ok] <= np.broadcast_to(tol, y.shape)[ok]).all(), np.max((np.abs(got - y) / tol)[ok])
        ok = np.isfinite(S)
        np.testing.assert_array_equal(np.isfinite(state), ok)
        assert (np.abs(state - S)[ok] <= np.broadcast_to(tol[:, None], S.shape)[ok]).all()


@pytest.mark.parametrize("heads,groups,dv,lens,head_decay,lo", [
    (2, 2, 64, [16], False, 0.5), (4, 2, 64, [31, 1, 64], False, 0.9), (8, 1, 64, [17, 97], True, 0.5), (3, 3, 128, [33, 130], False, 0.02), (2, 1, 192, [65, 40], True, 0.99)])
def test_delta_prompts_and_portions(cuda, heads, groups, dv, lens, head_decay, lo):
    """Chunk edges and tails, single tokens beside prompts, decays from next to nothing to next to one, a second portion that goes on from the slots."""
    rng = np.random.default_rng(sum(lens) + dv)
    state = torch.full((len(lens), heads, DK, dv), 7.0, device=cuda)
    S = [np.zeros((heads, DK, dv))] * len(lens)
    for portion in range(2):
        seqs = [_delta_seq(rng, n, heads, groups, dv, head_decay, lo) for n in lens]
        ys = _delta_run(cuda, seqs, heads, groups, dv, state, [portion * n for n in lens], head_decay)
        st = state.cpu().numpy()
        for i, (q, y) in enumerate(zip(seqs, ys)):
            _delta_check(q, S[i], y, st[i], heads, groups, lens[i])
        S = [st[i].astype(np.float64) for i in range(len(lens))]


@pytest.mark.parametrize("what", ["v nan", "v inf", "k nan", "q inf", "g zero", "g above one", "g nan", "beta nan", "k large", "all zero"])
def test_delta_odd_values(cuda, what):
    heads, groups, dv, n, at = 4, 2, 64, 60, 21
    rng = np.random.default_rng(9)
    seqs = [_delta_seq(rng, n, heads, groups, dv, False), _delta_seq(rng, n, heads, groups, dv, False)]
    s = seqs[0]
    if what == "v nan": s["v"][at, 1, 5] = np.nan
    elif what == "v inf": s["v"][at, 1, 5] = np.inf
    elif what == "k nan": s["k"][at, 0, 3] = np.nan
    elif what == "q inf": s["q"][at, 1, 9] = np.inf
    elif what == "g zero": s["g"][at] = 0.0
    elif what == "g above one": s["g"][at] = 1.25
    elif what == "g nan": s["g"][at, 2, 7] = np.nan
    elif what == "beta nan": s["b"][at, 0] = np.nan
    elif what == "k large": s["k"][n - 1] *= np.float32(2.0 ** 40)
    else:
        for x in "qkv": s[x][:] = 0.0
    state = torch.zeros((2, heads, DK, dv), device=cuda)
    ys = _delta_run(cuda, seqs, heads, groups, dv, state, [0, 0], False)
    st = state.cpu().numpy()
    for i in range(2):
        _delta_check(seqs[i], np.zeros((heads, DK, dv)), ys[i], st[i], heads, groups, n)
