"""silu of every bf16 value, as the GEMM epilogues and the activation kernel form it."""
import pytest
import torch


@pytest.mark.gpu
def test_silu_of_every_bf16_value_is_rounded_right(cuda):
    """Beside up = 1 the activation is silu(g) alone, rounded to bf16: half a unit in the last place (2^-8 at the most) and what f32 adds to it: an
    exponential of |g| log2(e) rounded to f32 (|g| 2^-24 and 2 units), a sum and a quotient, within (|g| + 4) 2^-23.  Below -88.72 e^-g overflows f32: -0, as g / (1 + e^-g) gives."""
    from nano_vllm_rs_b200 import ops
    g = torch.arange(65536, dtype=torch.int32, device="cuda").to(torch.int16).view(torch.bfloat16)
    got = ops.silu_mul(torch.cat([g, torch.ones_like(g)])[None])[0].double()
    x = g.double()
    ref = x / (1 + torch.exp(-x))
    normal = (x > -88.72) & x.isfinite() & (ref.abs() > 2.0 ** -126)
    err = (got - ref).abs() / ref.abs()
    worst = (err / (2.0 ** -8 + (x.abs() + 4) * 2.0 ** -23)).masked_fill(~normal, 0.0)
    assert float(worst.max()) <= 1, (float(worst.max()), float(x[worst.argmax()]), float(got[worst.argmax()]))
    assert (got[(x < -88.8) & x.isfinite()] == 0).all() and got[x == float("inf")].item() == float("inf")
    assert got[x.isnan()].isnan().all() and got[x == float("-inf")].isnan().all() and (got[x == 0] == 0).all()


@pytest.mark.gpu
def test_silu_of_every_bf16_value_is_that_of_the_quotient_to_the_bit(cuda):
    """g / (1 + e^-g) in f32 with the exponential of the math library and a division that rounds right, then rounded to bf16: the same 65536 results."""
    from nano_vllm_rs_b200 import ops
    g = torch.arange(65536, dtype=torch.int32, device="cuda").to(torch.int16).view(torch.bfloat16)
    got = ops.silu_mul(torch.cat([g, torch.ones_like(g)])[None])[0]
    want = (g.float() / (1 + torch.exp(-g.float()))).to(torch.bfloat16)
    number = ~want.isnan()
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got[number].view(torch.int16), want[number].view(torch.int16)), g[number][got[number].view(torch.int16) != want[number].view(torch.int16)]
