"""-m gpu test of the convolution's one-launch form (as many tokens as sequences): results and state against numpy."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _meta(lens, at, slots, cuda):
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=cuda)
    seq = np.repeat(np.arange(len(lens)), lens)
    pos = np.concatenate([np.arange(a, a + n) for a, n in zip(at, lens)])
    return i32(seq), i32(slots), i32(np.concatenate([[0], np.cumsum(lens)])), torch.from_numpy(pos).to(cuda)


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("ch", [4, 516, 1030])                       # one thread, a second CTA of one thread, a width for the general form
@pytest.mark.parametrize("lens", [[1] * 7, [2, 0, 1], [0, 0, 5, 0, 0]])
def test_as_many_tokens_as_sequences(cuda, taps, ch, lens):
    from nano_vllm_rs_b200 import ops
    rng = np.random.default_rng(taps + ch)
    n, H = len(lens), taps - 1
    at = [0, 1, 2, 3, 9, 700, 4][:n]                                 # some windows reach back before the sequence
    slots = [5, 0, 2, 7, 1, 3, 4][:n]
    if n == 7:
        slots[3] = -1                                                # a padding row: zeros, no state
    f = lambda *s: rng.standard_normal(s).astype(np.float32)
    x, w, b, st = f(n, ch + 4), f(ch, taps), f(ch), f(8, H, ch)
    state = torch.from_numpy(st).to(cuda)
    out = ops.causal_conv(torch.from_numpy(x).to(cuda)[:, :ch], torch.from_numpy(w).to(cuda), torch.from_numpy(b).to(cuda), state, *_meta(lens, at, slots, cuda))
    ref, new, o = np.zeros((n, ch)), st.astype(np.float64).copy(), 0
    for s, m in enumerate(lens):
        if slots[s] >= 0 and m:
            past = st[slots[s]].astype(np.float64).copy()
            past[:max(H - at[s], 0)] = 0
            row = np.vstack([past, x[o:o + m, :ch]])
            for t in range(m):
                ref[o + t] = (row[t:t + taps] * w.T).sum(0) + b
            new[slots[s]] = row[m:m + H]
        o += m
    silu = ref / (1 + np.exp(-ref))
    # up to five roundings of terms of a few units, then the quotient of the activation
    np.testing.assert_allclose(out.cpu().numpy(), silu, rtol=4e-6, atol=4e-6)
    np.testing.assert_array_equal(state.cpu().numpy(), new.astype(np.float32))
