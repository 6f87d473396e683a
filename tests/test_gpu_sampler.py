"""-m gpu parity tests for the device sampler (K12, nvllm_sample) against the oracle restatement of
Sampler::forward (sampler.rs:26-219, oracle/layers.py).

What is bit-exact: greedy tokens, the top-k survivor set (including the stable-sort tie rule), the uniforms of the
seeded contract.  What carries a stated tolerance: the top-p survivor set (the reference accumulates f32 probabilities
sequentially over ~150K entries — its own rounding error moves the cut; the kernel sums exactly in fixed point) and the
Gumbel-max winner (logf differs from numpy's log by an ulp): the kernel's token must score within 1e-4 of the oracle's
best score over the kernel's own survivor set."""
import numpy as np
import pytest
import torch

from oracle import layers as O

pytestmark = pytest.mark.gpu

TOP_P_MASS_TOL = 2e-4   # f32 sequential cumulative-sum error bound of the reference at V ~ 150K
SCORE_TOL = 1e-4


def run(cuda, logits, temps, seeds, top_k=None, top_p=None):
    from nano_vllm_rs_b200 import ops
    lg = torch.from_numpy(logits).to(cuda)
    t = torch.tensor(temps, dtype=torch.float32, device=cuda)
    sd = torch.from_numpy(np.asarray(seeds, dtype=np.uint64).view(np.int64)).to(cuda)
    tk = None if top_k is None else torch.tensor(top_k, dtype=torch.int32, device=cuda)
    tp = None if top_p is None else torch.tensor(top_p, dtype=torch.float32, device=cuda)
    ids, cnt, mask = ops.sample(lg, t, sd, top_k=tk, top_p=tp, debug=True)
    torch.cuda.synchronize()
    return ids.cpu().numpy(), cnt.cpu().numpy(), mask.cpu().numpy().astype(bool)


def check_token(logits_row, T, mask_row, seed, tok):
    """Gumbel-max over the kernel's own survivor set, oracle arithmetic."""
    s = logits_row / np.float32(T) if T != 1.0 else logits_row
    scores = np.where(mask_row, s + O.sample_gumbel(O.sampler_uniform(seed, len(s))), -np.inf)
    assert mask_row[tok], "sampled token is not in the survivor set"
    assert scores[tok] >= scores.max() - SCORE_TOL, (tok, int(scores.argmax()), scores[tok], scores.max())


def seeds_for(n, base=99):
    return [O.sampler_row_seed(base, i, 17 + i) for i in range(n)]


def test_greedy_rows_first_maximum(cuda):
    rng = np.random.default_rng(0)
    x = rng.standard_normal((6, 5000)).astype(np.float32)
    x[1, [7, 4000]] = 9.0          # tie: first index wins
    x[2, :] = 0.0                  # all equal -> 0
    x[3, 4999] = 50.0
    ids, cnt, mask = run(cuda, x, [0.0] * 6, seeds_for(6), top_k=[5] * 6, top_p=[0.5] * 6)   # filters ignored when T == 0
    assert ids.tolist() == np.argmax(x, -1).tolist() and ids[1] == 7 and ids[2] == 0
    assert (cnt == 5000).all() and mask.all()


@pytest.mark.parametrize("V", [1000, 151936])
def test_top_k_survivor_set_bit_exact(cuda, V):
    rng = np.random.default_rng(V)
    B = 7
    x = (rng.standard_normal((B, V)) * 3).astype(np.float32)
    x[5] = np.round(x[5])                       # heavy ties, some straddling k
    x[6] = 1.25                                 # everything ties: the first k indices survive
    temps = [1.0, 0.7, 1.3, 1.0, 2.0, 1.0, 0.5]
    ks = [1, 50, 4000 if V > 4000 else 400, V, V + 5, 37, 10]
    seeds = seeds_for(B)
    ids, cnt, mask = run(cuda, x, temps, seeds, top_k=ks)
    for b in range(B):
        _, filt, _ = O.sample_single(x[b], temps[b], None, ks[b], seeds[b])
        want = np.isfinite(filt)
        assert cnt[b] == want.sum() == min(ks[b], V)
        assert (mask[b] == want).all(), f"row {b}: top-k set differs in {(mask[b] != want).sum()} places"
        check_token(x[b], temps[b], mask[b], seeds[b], ids[b])
    assert mask[6, :10].all() and not mask[6, 10:].any()


def check_top_p_set(s, mask_row, p):
    """mask must be a prefix of the descending order whose exact (f64) mass reaches p, minimal up to the tolerance."""
    e = np.exp(s.astype(np.float64) - s.max())
    prob = e / e.sum()
    kept, drop = prob[mask_row], prob[~mask_row]
    assert kept.size >= 1
    if drop.size:
        assert kept.min() >= drop.max() * (1 - 1e-6), "survivors are not a prefix of the descending order"
    mass = kept.sum()
    assert mass >= p - TOP_P_MASS_TOL, (mass, p)
    assert mass - kept.min() < p + TOP_P_MASS_TOL, (mass, kept.min(), p)   # dropping the smallest survivor falls below p


@pytest.mark.parametrize("V", [2000, 151936])
def test_top_p_survivor_set(cuda, V):
    rng = np.random.default_rng(V + 1)
    B = 6
    x = (rng.standard_normal((B, V)) * np.array([1, 2, 4, 6, 0.02, 3])[:, None]).astype(np.float32)
    temps = [1.0, 0.8, 1.0, 1.5, 1.0, 1.0]
    ps = [0.9, 0.5, 0.95, 0.1, 0.3, 1.0]       # 1.0 = None
    seeds = seeds_for(B, 5)
    ids, cnt, mask = run(cuda, x, temps, seeds, top_p=ps)
    for b in range(B):
        s = x[b] / np.float32(temps[b]) if temps[b] != 1.0 else x[b]
        if ps[b] >= 1.0:
            assert mask[b].all()
        else:
            check_top_p_set(s, mask[b], ps[b])
            # and the oracle's own cut (f32 sequential cumsum) is within the same tolerance of ours
            _, filt, _ = O.sample_single(x[b], temps[b], ps[b], None, seeds[b])
            e = np.exp(s.astype(np.float64) - s.max()); prob = e / e.sum()
            assert abs(prob[np.isfinite(filt)].sum() - prob[mask[b]].sum()) <= 2 * TOP_P_MASS_TOL + prob.max()
        assert cnt[b] == mask[b].sum()
        check_token(x[b], temps[b], mask[b], seeds[b], ids[b])


def test_top_k_then_top_p_and_ties(cuda):
    rng = np.random.default_rng(3)
    V, B = 4096, 5
    x = (rng.standard_normal((B, V)) * 2).astype(np.float32)
    x[3] = np.round(x[3] * 2) / 2               # tie groups at the top-p cut
    x[4] = 0.5                                  # uniform: top-k 100 then top-p 0.25 -> first 25 indices
    temps, ks, ps = [1.0, 0.6, 1.2, 1.0, 1.0], [50, 200, 0, 300, 100], [0.8, 0.9, 0.7, 0.6, 0.25]
    seeds = seeds_for(B, 8)
    ids, cnt, mask = run(cuda, x, temps, seeds, top_k=ks, top_p=ps)
    for b in range(B):
        s = x[b] / np.float32(temps[b]) if temps[b] != 1.0 else x[b].copy()
        if ks[b]:
            s = O.apply_top_k(s, ks[b])
        fin = np.isfinite(s)
        assert not mask[b][~fin].any()
        check_top_p_set(np.where(fin, s, -np.inf)[fin], mask[b][fin], ps[b])
        check_token(x[b], temps[b], mask[b], seeds[b], ids[b])
    assert mask[4, :25].all() and cnt[4] == 25
    # whole pipeline vs the oracle where no tolerance is involved (peaked rows: the cut is far from any rounding)
    for b in (0, 1):
        want = O.sampler_forward(x[b:b + 1], temps[b:b + 1], ps[b:b + 1], ks[b:b + 1], seeds[b:b + 1])[0]
        _, _, scores = O.sample_single(x[b], temps[b], ps[b], ks[b], seeds[b])
        assert ids[b] == want or scores[ids[b]] >= scores.max() - SCORE_TOL


def test_seeded_contract_determinism_and_distribution(cuda):
    V, B = 8, 8192
    row = np.array([2.0, 1.0, 0.5, 0.0, -0.5, -1.0, 1.5, -3.0], dtype=np.float32)
    x = np.tile(row, (B, 1))
    seeds = [O.sampler_row_seed(1234, i, 3) for i in range(B)]
    ids1, _, _ = run(cuda, x, [1.0] * B, seeds)
    ids2, _, _ = run(cuda, x, [1.0] * B, seeds)
    assert (ids1 == ids2).all()
    want = O.sampler_forward(x, [1.0] * B, None, None, seeds)
    assert (ids1 == want).mean() > 0.999           # only logf-ulp near-ties may differ
    freq = np.bincount(ids1, minlength=V) / B
    prob = np.exp(row - row.max()); prob /= prob.sum()
    assert np.abs(freq - prob).max() < 0.02, (freq, prob)   # Gumbel-max samples the softmax
    ids3, _, _ = run(cuda, x, [1.0] * B, [O.sampler_row_seed(1235, i, 3) for i in range(B)])
    assert (ids3 != ids1).mean() > 0.3


@pytest.mark.parametrize("V", [1000, 20001, 70000, 151936])   # 20001: rows off 16 bytes
def test_short_cuts_select_what_the_radix_selection_selects(cuda, V):
    """Logits and temperature times 2^24 give the same scaled values to the bit, but lie beyond the range of temperatures that the
    candidate and linear-bin short cuts take: survivors and tokens have to be identical."""
    rng = np.random.default_rng(V)
    combos = [(k, p) for k in (0, 1, 50, 255, 256, 257) for p in (0.0, 0.1, 0.9, 0.999)]
    B = len(combos)
    x = (rng.standard_normal((B, V)) * 3).astype(np.float32)
    x[::3] = np.round(x[::3] * 4) / 4           # tie groups at both cuts
    x[1::6] = np.sort(x[1::6], -1)              # the largest values in one place
    x[4, : V // 2] = -np.inf
    x[5, 3] = np.nan                            # left to the radix selection
    x[7] = 0.5
    temps = (0.4 + 0.1 * np.arange(B)).astype(np.float32)
    ks, ps = [k for k, _ in combos], [p for _, p in combos]
    seeds = seeds_for(B, 21)
    a = run(cuda, x, temps, seeds, top_k=ks, top_p=ps)
    b = run(cuda, x * np.float32(2 ** 24), temps * np.float32(2 ** 24), seeds, top_k=ks, top_p=ps)
    for got, want in zip(a, b):
        assert (got == want).all()


@pytest.mark.parametrize("top", [3.0, 25.0, 100.0, 150.0, -150.0])
def test_masses_of_large_scaled_values(cuda, top):
    """At a temperature of 1e-6 neighbouring logits lie whole units apart: 100 000 values some steps below the maximum have a mass (one of
    2^32 at 22 below) that decides the cut.  Times 2^44 the same scaled values go to the radix selection."""
    V = 120000
    steps = [1, 2, 3, 5, 6, 7, 11, 12, 23, 90, 180]
    ps = [0.5, 0.995, 0.99999]
    rows = []
    for s in steps:
        x = np.full(V, top - 1.0, np.float32)
        below = np.float32(top)
        for _ in range(s):
            below = np.nextafter(below, np.float32(-np.inf), dtype=np.float32)
        x[10:100010] = below
        x[7] = top
        rows.append(x)
    x = np.repeat(np.stack(rows), len(ps), 0)
    B = len(x)
    top_p, temps, seeds = ps * len(steps), np.full(B, 1e-6, np.float32), seeds_for(B, 5)
    a = run(cuda, x, temps, seeds, top_p=top_p)
    b = run(cuda, x * np.float32(2.0 ** 44), temps * np.float32(2.0 ** 44), seeds, top_p=top_p)
    for got, want in zip(a, b):
        assert (got == want).all()


@pytest.mark.parametrize("rows", [24, 168])        # 1024 threads a row, and 512 beyond one row per SM
@pytest.mark.parametrize("V", [4096, 20001, 151936])
def test_tokens_do_not_depend_on_what_else_is_asked_for(cuda, rows, V):
    """Without the survivors' count and mask, a value that cannot win is skipped before its noise is computed: the tokens are the same."""
    from nano_vllm_rs_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(V + rows)
    x = 2.5 * torch.randn((rows, V), generator=g, device=cuda)
    T = torch.tensor([0.1, 0.5, 1.0, 1.7, 3.0, 0.0], device=cuda).repeat(rows // 6)
    x[1::12] *= 400.0                                      # quotients on both sides of 1e4, where the skip ends
    x[2::12] = torch.round(x[2::12])                       # ties
    x[3::24] = x[3::24].sort(-1).values                    # the winner comes last
    x[4::24] = x[4::24].sort(-1, descending=True).values
    x[7::24, : V // 2] = float("-inf")
    x[8::24, 5] = float("inf")
    x[9::24, 3] = float("nan")
    x[10::24, 100:200] = float("nan")                      # with top-k 50 every survivor is NaN
    x[13::24] = float("nan")
    x[14::24] = float("-inf")
    T[13::24], T[15::24] = 1e-6, 1e6
    seeds = torch.randint(-(1 << 62), 1 << 62, (rows,), generator=g, device=cuda)
    for k, p in ((None, None), (50, None), (300, None), (None, 0.9), (300, 0.9), (50, 0.9)):
        tk = None if k is None else torch.full((rows,), k, dtype=torch.int32, device=cuda)
        tp = None if p is None else torch.full((rows,), p, device=cuda)
        ids, _, _ = ops.sample(x, T, seeds, tk, tp, debug=True)
        assert torch.equal(ids, ops.sample(x, T, seeds, tk, tp)), (k, p)


@pytest.mark.parametrize("V", [3000, 20000, 151936])
def test_top_k_of_values_close_to_one_another(cuda, V):
    """Rows whose largest values differ by less than 2^-11 of themselves (the bound of the candidates then takes all 32 bits), on either side of it, and tied."""
    rng = np.random.default_rng(V + 7)
    spread = np.array([1e-2, 1e-3, 1e-4, 3e-6, 1e-2, 0.3])[:, None]
    x = (np.array([10, 10, -10, 10, 1e4, 10])[:, None] + rng.standard_normal((6, V)) * spread).astype(np.float32)
    temps, ks, seeds = [1.0, 0.8, 1.0, 1.0, 0.9, 1.0], [1, 50, 20, 200, 256, 9], seeds_for(6, 13)
    ids, cnt, mask = run(cuda, x, temps, seeds, top_k=ks)
    for b in range(6):
        want = np.isfinite(O.sample_single(x[b], temps[b], None, ks[b], seeds[b])[1])
        assert cnt[b] == want.sum() == ks[b] and (mask[b] == want).all()
        check_token(x[b], temps[b], mask[b], seeds[b], ids[b])
