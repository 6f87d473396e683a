"""Epilogues write 32 bytes at once where the rows of the output lie on 32 bytes, and by 16 elsewhere: the same bits, and nothing beside them."""
import pytest
import torch


def views(rows, cols, dtype):
    """Outputs inside a larger buffer: rows on 32 bytes; a start, and for bf16 a pitch (of 8 values, as ever), that are odd multiples of 16 bytes."""
    step = 16 // torch.empty(0, dtype=dtype).element_size()
    for at, pitch in ((0, 16), (step, 16), (0, 24), (3 * step, 8)):
        ld = (cols + 15) // 16 * 16 + pitch
        buf = torch.full((rows + 1, ld), 777.0, dtype=dtype, device="cuda")
        yield buf, buf.view(-1)[at:at + rows * ld].view(rows, ld)[:, :cols]


def check(run, rows, cols, dtype):
    want = run(torch.empty(rows, cols, dtype=dtype, device="cuda"))
    assert torch.isfinite(want.float()).all()
    for buf, out in views(rows, cols, dtype):
        got = run(out).clone()
        assert torch.equal(got, want)
        out.fill_(777.0)
        assert bool((buf == 777.0).all())


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(1, 136, 64), (128, 264, 128), (129, 72, 64), (300, 264, 192), (513, 2056, 64), (2600, 4104, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_products(cuda, m, n, k, dtype):
    from nano_vllm_rs_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16)
    w = torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16)
    check(lambda y: ops.gemm_bf16(x, w, out=y), m, n, dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("m,inter", [(100, 128), (300, 384), (2600, 1536)])
def test_gated_products(cuda, m, inter):
    from nano_vllm_rs_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn(m, 64, generator=gen, device="cuda").to(torch.bfloat16)
    w = torch.randn(2 * inter, 64, generator=gen, device="cuda").to(torch.bfloat16)
    check(lambda y: ops.gemm_silu_mul(x, w, out=y), m, inter, torch.bfloat16)


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [(1, 130), (257,)])
def test_prompt_attention(cuda, lens):
    from nano_vllm_rs_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(len(lens))
    n, H, G, D = sum(lens), 4, 2, 128
    q, k, v = (torch.randn(n, h, D, generator=gen, device="cuda").to(torch.bfloat16) for h in (H, G, G))
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device="cuda")
    check(lambda y: ops.varlen_prefill_attention(q, k, v, cu, cu, max(lens), max(lens), out=y), n, H * D, torch.bfloat16)
