"""-m gpu test of the sort of assignments by expert, by one CTA and by a cluster, against numpy."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,top,experts,spread", [(1023, 2, 64, 64), (1024, 2, 64, 64), (5000, 3, 7, 7), (1500, 2, 1024, 1024), (1500, 2, 1025, 1025),
                                                  (40, 2, 6143, 6143), (4096, 1, 64, 1), (1100, 2, 33, 48)])   # one expert takes all; identity experts
@pytest.mark.parametrize("tile", [32, 128])
def test_expert_sort(cuda, n, top, experts, spread, tile):
    from nano_vllm_rs_b200 import ops
    idx = torch.randint(0, spread, (n, top), generator=torch.Generator().manual_seed(n), dtype=torch.int32)
    wts = torch.rand(n, top, generator=torch.Generator().manual_seed(n + 1))
    row_token, row_w, tile_expert, slot_row = [t.cpu().numpy() for t in ops.moe_sort_weighted(idx.to(cuda), wts.to(cuda), experts, tile_rows=tile)]
    flat, slot = idx.numpy().reshape(-1), slot_row.reshape(-1)
    live = flat < experts
    assert (slot[~live] == -1).all() and len(set(slot[live])) == live.sum()
    rows = slot[live]
    assert np.array_equal(tile_expert[rows // tile], flat[live]) and np.array_equal(row_token[rows], np.nonzero(live)[0] // top)
    assert np.array_equal(row_w[rows], wts.numpy().reshape(-1)[live])
    pad = np.ones(len(row_token), bool); pad[rows] = False
    assert (row_token[pad] == -1).all() and (row_w[pad] == 0).all()
    tiles = -(-np.bincount(flat[live], minlength=experts) // tile)                                             # experts in order, no tile spare
    assert np.array_equal(tile_expert, np.concatenate([np.repeat(np.arange(experts), tiles), np.full(len(tile_expert) - tiles.sum(), -1)]))
