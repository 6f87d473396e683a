"""-m gpu tests of the vectorised passes over a prompt's rows, at the edges of their rules, against plain PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("with_res", [False, True])
@pytest.mark.parametrize("hidden", [8, 264, 1016, 1024, 1032])      # one piece, ragged and full lanes, the first width past the rule
@pytest.mark.parametrize("rows", [2367, 2368, 2373])                # 16 rows per SM of 148: below, at, and with a last CTA of 5 rows
def test_rms_norm_of_many_rows(cuda, rows, hidden, with_res):
    from nano_vllm_rs_b200 import ops
    g = torch.Generator().manual_seed(rows + hidden)
    x, res = [torch.randn(rows, hidden, generator=g).bfloat16() for _ in range(2)]
    w = (1 + 0.1 * torch.randn(hidden, generator=g)).bfloat16()
    rd = res.to(cuda) if with_res else None
    got = ops.add_rmsnorm(x.to(cuda), w.to(cuda), 1e-6, residual=rd).cpu().double()
    s = (x.float() + res.float()).bfloat16() if with_res else x
    if with_res:
        assert torch.equal(rd.cpu(), s)
    s = s.double()
    ref = s / (s.square().mean(1, keepdim=True) + 1e-6).sqrt() * w.double()
    assert ((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-30).all()   # one rounding to bf16 (half an ulp: 2^-9) and f32's noise before it


@pytest.mark.parametrize("dims,scale", [(128, 1.0), (64, 0.5), (64, 1.0), (8, 0.25), (124, 0.5)])   # 124: not in fours of pairs
@pytest.mark.parametrize("n", [147, 148, 300])
@pytest.mark.parametrize("offset", [0, 4, 1])                                                      # 1: rows that no 16-byte load can read
def test_rotate_half_of_many_tokens(cuda, n, dims, scale, offset):
    from nano_vllm_rs_b200 import ops
    H, dim = 5, 128
    g = torch.Generator().manual_seed(n + dims)
    x = torch.randn(n, H * dim + 8, generator=g)
    pos = torch.randint(0, 700, (n,), generator=g)
    tab = ops.rope_table_interleaved(600, dims, 1e4, cuda)           # positions past the table take its last row
    xd = x.to(cuda)
    ops.rotate_half(xd[:, offset:], pos.to(cuda), tab, H, dim, dims, scale)
    cs = tab.cpu().double().reshape(600, dims // 2, 2)[pos.clamp(max=599)][:, None]
    v = x[:, offset:offset + H * dim].double().reshape(n, H, dim)
    u, w = v[..., :dims // 2], v[..., dims // 2:dims]
    ref = torch.cat([u * cs[..., 0] - w * cs[..., 1], w * cs[..., 0] + u * cs[..., 1], v[..., dims:]], -1) * scale
    got = xd.cpu()
    tol = 3 * 2.0 ** -24 * scale * (u.abs() + w.abs()).max()         # two products and a sum, each rounded once
    assert (got[:, offset:offset + H * dim].reshape(n, H, dim).double() - ref).abs().max() <= tol
    rest = torch.ones(x.shape[1], dtype=torch.bool); rest[offset:offset + H * dim] = False
    assert torch.equal(got[:, rest], x[:, rest])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hidden", [4, 6, 1028, 2048])
def test_scaled_embedding_rows(cuda, hidden, dtype):
    from nano_vllm_rs_b200 import ops
    g = torch.Generator().manual_seed(hidden)
    table = torch.randn(37, hidden, generator=g).to(dtype)
    ids = torch.tensor([0, 36, 5, 5, -1, 37, 1 << 40])               # out of range: the nearest row
    h, h2 = ops.embedding_gather_scaled(table.to(cuda), ids.to(cuda), 2.5, copy=True)
    assert torch.equal(h.cpu(), table[ids.clamp(0, 36)].float() * 2.5) and torch.equal(h, h2)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("q,k,v", [(1024, 256, 128), (8, 4, 12), (8, 6, 4)])
@pytest.mark.parametrize("which", [(1, 1, 1), (0, 1, 0), (1, 0, 1)])
def test_store_with_some_biases(cuda, q, k, v, which, dtype):
    from nano_vllm_rs_b200 import ops
    n = 9
    g = torch.Generator().manual_seed(q + k)
    proj = torch.randn(n, q + k + v, generator=g)
    bias = [torch.randn(c, generator=g) if on else None for c, on in zip((q, k, v), which)]
    dev = lambda b: None if b is None else b.to(cuda)
    kc, vc = torch.zeros(20, k, dtype=dtype, device=cuda), torch.zeros(20, v, dtype=dtype, device=cuda)
    slots = torch.tensor([3, 19, -1, 0, 7, 8, -1, 1, 2], dtype=torch.int32)
    got = ops.attn_bias_store(proj.to(cuda), q, k, v, *[dev(b) for b in bias], kc, vc, slots.to(cuda), dtype)
    want = [p + b if b is not None else p for p, b in zip(proj.split([q, k, v], 1), bias)]
    live = slots >= 0
    for cache, w in ((kc, want[1]), (vc, want[2])):
        ref = torch.zeros(20, w.shape[1]); ref[slots[live].long()] = w[live]
        assert torch.equal(cache.cpu(), ref.to(dtype))
    assert torch.equal(got.cpu(), want[0].to(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("gs", [4, 100, 128, 132])                                                 # up to 128: four parts a warp
@pytest.mark.parametrize("rows,parts", [(18943, 1), (18945, 1), (1723, 11)])                       # 128 parts per SM of 148; last warps of 1 and 3 parts
@pytest.mark.parametrize("gate_first", [False, True])
def test_gated_norm_of_many_parts(cuda, rows, parts, gs, gate_first, dtype):
    from nano_vllm_rs_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(rows + gs)
    y, z = [torch.randn(rows, parts * gs, generator=g, device=cuda) for _ in range(2)]
    w = 1 + 0.1 * torch.randn(parts * gs, generator=g, device=cuda)
    got = ops.gated_group_norm(y, z, w, parts, 1e-5, gate_first, dtype).double()
    s = torch.nn.functional.silu(z.double())
    v = (y.double() * s if gate_first else y.double()).reshape(rows, parts, gs)
    ref = (v / (v.square().mean(-1, keepdim=True) + 1e-5).sqrt()).reshape(rows, -1) * (1 if gate_first else s) * w.double()
    tol = 2e-6 + (2.0 ** -8 if dtype == torch.bfloat16 else 0)      # expf and a quotient (3 ulp), rsqrtf (2), the sum and four products: 16 * 2^-23
    assert ((got - ref).abs() <= tol * ref.abs() + 1e-30).all()


@pytest.mark.parametrize("n", [1, 592, 593])                                                       # up to four tokens per SM of 148: two CTAs a token
def test_delta_preparation(cuda, n):
    from nano_vllm_rs_b200 import ops
    H, G, D = 3, 2, 128
    g = torch.Generator(device=cuda).manual_seed(n)
    rn = lambda *s: torch.randn(*s, generator=g, device=cuda)
    q, k, beta, raw, alog, bias = rn(n, G * D), rn(n, G * D), rn(n, H), 2 * rn(n, H * D), rn(H), rn(H * D)
    want = []
    for x, scale in ((q, 0.5), (k, 1.0)):
        v = x.double().reshape(n, G, D)
        want.append((v * scale / (v.square().sum(-1, keepdim=True) + 1e-6).sqrt()).reshape(n, -1))
    want.append(beta.double().sigmoid())
    want.append((-alog.double().exp().repeat_interleave(D) * torch.nn.functional.softplus(raw.double() + bias.double())).exp())
    ops.delta_prepare(q, k, beta, raw, alog, bias, H, G, D, 0.5)
    for got, ref in zip((q, k, beta, raw), want):
        # unit vectors and sigmoids: a few roundings each; a decay exp(-x) has x's relative error (8 * 2^-24) times x, at most 745
        assert ((got.double() - ref).abs() <= 2e-6 * ref.abs() * (1 + ref.abs().clamp(min=1e-300).log().abs()) + 1e-37).all()
