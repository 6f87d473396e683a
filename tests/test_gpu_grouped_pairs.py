"""-m gpu test of the experts' product on CTA pairs (two neighbouring 128-row tiles of one group) against float64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(248, 64), (256, 64), (264, 192), (520, 1408)])          # below the pairs' width, at it, ragged last tiles
@pytest.mark.parametrize("runs", [[(0, 4)], [(2, 1), (0, 1), (1, 1), (2, 1)], [(0, 3), (-1, 1), (0, 2), (3, 5), (1, 1)], [(-1, 4)],
                                  [(3, 31), (0, 2), (2, 32), (1, 33), (0, 1), (-1, 6)]])   # runs across the list's blocks of 32
@pytest.mark.parametrize("relu2", [False, True])
def test_every_tile_takes_its_own_group(cuda, runs, n, k, relu2):
    from nano_vllm_rs_b200 import _ffi, ops
    group = np.concatenate([np.full(c, g, np.int32) for g, c in runs])
    rows = 128 * len(group)
    gen = torch.Generator(device=cuda).manual_seed(n + k + rows)
    x = torch.randn(rows, k + 8, generator=gen, device=cuda).bfloat16()[:, :k]
    w = torch.randn(4 * n, k, generator=gen, device=cuda).bfloat16()
    y = torch.full((rows + 128, n + 8), 7.0, device=cuda, dtype=torch.bfloat16)            # a strip beside and a tile below that nothing writes
    tiles = torch.from_numpy(group).to(cuda)
    call = _ffi.lib().nvllm_gemm_relu2_bf16_grouped if relu2 else _ffi.lib().nvllm_gemm_bf16_grouped
    _ffi.check(call(y.data_ptr(), x.data_ptr(), w.data_ptr(), rows, n, k, 4, x.stride(0), k, y.stride(0), tiles.data_ptr(),
                                                  torch.cuda.current_stream().cuda_stream))
    assert (y[rows:] == 7).all() and (y[:, n:] == 7).all()
    live = tiles.repeat_interleave(128) >= 0
    wg = w.double().reshape(4, n, k)
    for g in range(4):
        on = tiles.repeat_interleave(128) == g
        a = x[on].double()
        ref, size = a @ wg[g].T, a.abs() @ wg[g].abs().T
        tol = 2.0 ** -8 * ref.abs() + k * 2.0 ** -24 * size                                 # the product's rounding to bf16; f32 sums
        if relu2:                                                                           # (v + t)^2 - v^2, and a second rounding
            tol, ref = 2.1 * tol * ref.abs() + tol ** 2 + 2.0 ** -8 * ref.square(), ref.clamp(min=0).square()
        assert ((y[:rows][on][:, :n].double() - ref).abs() <= tol).all()
    assert torch.isfinite(y[:rows][live].float()).all()
