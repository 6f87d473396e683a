"""Products of prompts: the order of their tiles, and the ones that add to the residual stream."""
import numpy as np
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(4200, 3400, 3072), (3841, 4352, 3072), (700, 1800, 3072), (1025, 776, 4096), (4400, 264, 3136)])
def test_panels_of_tiles_cover_the_product(cuda, m, n, k):
    """Panels of 12 n-tiles (16 m-tiles and more) and of 2, with a narrower last panel, one panel alone, and ragged edges: f32 sums in another
    order than the check kernel's."""
    from nano_vllm_rs_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16)
    w = (torch.randn(n, k, generator=gen, device="cuda") * 0.02).to(torch.bfloat16)
    y, r = (ops.gemm_bf16(x, w, out_dtype=torch.float32, simt=s) for s in (False, True))
    assert float((y - r).abs().max()) < 3e-3 and float((y - r).norm() / r.norm()) < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(6200, 3400, 3072), (4200, 3400, 8192), (6200, 2056, 3072), (4200, 1032, 1024)])
def test_panels_by_the_length_of_the_rows(cuda, m, n, k):
    """Panels of 12 from 24 m-tiles on, and from 16 on where rows are long, with a narrower last one; rows of the product that do not lie on 32 bytes; no panels."""
    test_panels_of_tiles_cover_the_product(cuda, m, n, k)


@pytest.mark.gpu
def test_prompts_give_the_same_logits_where_projections_add_to_the_stream(cuda):
    """Together the prompts have more tiles than pairs, and their o / down projections add to the stream; either half of them, on the same
    kernels otherwise, goes through the separate add.  Both round in the same places."""
    from nano_vllm_rs_b200 import engine as E
    rng = np.random.default_rng(5)
    prompts = [rng.integers(0, 512, int(n)) for n in [512, 511, 700, 300, 640, 1000, 257, 256, 301, 423]]
    total = sum(len(p) for p in prompts)
    assert total > 18 * 256 and 512 < sum(len(p) for p in prompts[5:]) < 18 * 256 > sum(len(p) for p in prompts[:5])

    def logits(groups):
        out = []
        for g in groups:
            eng = E.LLMEngine(E.Config("qwen3-0.6b", vocab_size=512, num_hidden_layers=2, max_num_seqs=len(prompts), max_num_batched_tokens=total,
                                       max_model_len=1024, kvcache_block_size=256, num_kvcache_blocks=40), seed=3, std=0.02)
            for p in g:
                eng.add_request(p, E.SamplingParams(temperature=0.0, max_tokens=4, ignore_eos=True))
            batch = eng.scheduler.schedule()
            assert batch.is_prefill and batch.c.num_seqs == len(g)
            out.append(eng.model_runner.execute_model(batch, return_logits=True)[1])
        return np.concatenate(out)
    assert np.array_equal(logits([prompts]), logits([prompts[:5], prompts[5:]]))


@pytest.mark.gpu
@pytest.mark.parametrize("width", [64, 128, 256])
def test_projections_add_to_the_stream_at_every_tile_width(cuda, width, monkeypatch):
    """The 4900 tokens above take tiles 128 wide by themselves, large prompts 256."""
    monkeypatch.setenv("NVLLM_GEMM_BN", str(width))
    test_prompts_give_the_same_logits_where_projections_add_to_the_stream(cuda)
