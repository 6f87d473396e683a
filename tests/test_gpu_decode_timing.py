"""Timing the decode attention and replaying a decode step behind the runner's back: the caches and the coming steps do not notice."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
VOCAB, LAYERS = 512, 3


def caches(runner):
    """Copies of every layer's keys and values."""
    import torch
    from nano_vllm_rs_b200 import _ffi
    out = []
    for l in range(LAYERS):
        k, v, lay = C.c_void_p(), C.c_void_p(), _ffi.KvLayout()
        _ffi.check(_ffi.lib().nvllm_runner_kv_cache(runner.h, l, C.byref(k), C.byref(v), C.byref(lay)))
        for p in (k, v):
            view = type("View", (), {"__cuda_array_interface__": {"shape": (runner.config.num_kvcache_blocks * lay.block_stride,), "typestr": "<i2", "version": 3,
                                                                  "data": (p.value, False)}})()
            out.append(torch.as_tensor(view, device="cuda").clone())
    return out


@pytest.mark.parametrize("seqs", [1, 3, 20])   # one token in one launch; few tokens, whose attention stores their keys itself; more
def test_timing_the_decode_attention_stores_nothing(cuda, seqs):
    """The rows that the projections left belong to the last layer, or to no step at all: stored again, they would be other layers' keys."""
    import torch
    from nano_vllm_rs_b200 import engine as E
    prompts = [np.random.default_rng(i).integers(0, VOCAB, 30 + 7 * i).tolist() for i in range(seqs)]

    def steps(time_between):
        cfg = E.Config("qwen3-0.6b", vocab_size=VOCAB, num_hidden_layers=LAYERS, max_num_seqs=seqs, max_num_batched_tokens=4096, max_model_len=512, kvcache_block_size=16,
                       num_kvcache_blocks=16 * seqs).validate()
        sched, runner = E.Scheduler(cfg), E.ModelRunner(cfg)
        runner.init_weights(7, 0.02)
        for p in prompts:
            sched.add_sequence(p, E.SamplingParams(temperature=0.0, max_tokens=8, ignore_eos=True))
        out = []
        while not sched.is_finished():
            b = sched.schedule()
            toks, logits = runner.execute_model(b, return_logits=True)
            out.append(logits)
            sched.postprocess(toks)
            if time_between and not b.is_prefill:
                before = caches(runner)
                ms, nbytes = runner.time_decode_attention(4)
                assert ms > 0 and nbytes > 0
                assert all(torch.equal(x, y) for x, y in zip(before, caches(runner)))
        return np.stack(out)

    assert np.array_equal(steps(True), steps(False))
