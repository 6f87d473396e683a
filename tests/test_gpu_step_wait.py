"""A decode step of one token in one launch whose thread blocks wait for a word that nobody writes."""
import numpy as np
import pytest

from tests.test_gpu_step_single import VOCAB, Decoder, weights_of

pytestmark = pytest.mark.gpu
DIMS = (1024, 16, 8, 3072)


@pytest.mark.parametrize("eager", [0, 1])
@pytest.mark.parametrize("silent", [0, 147])
@pytest.mark.parametrize("where", ["execute", "replay"])
def test_a_word_that_never_comes_is_the_error_of_that_step_alone(cuda, where, silent, eager):
    """The kernel ends by itself once the limit is over, whoever launched the step reports it, and the same step executed again, and the ones behind it, give
    what they give elsewhere: the words of the step that gave up are no other step's."""
    from nano_vllm_rs_b200 import _ffi, engine as E
    rng = np.random.default_rng(silent)
    weights, prompt, forced = weights_of(*DIMS, cuda), rng.integers(0, VOCAB, 70).tolist(), rng.integers(0, VOCAB, 8)
    want = Decoder(*DIMS, weights, 16, eager=eager).run(prompt, forced)
    d = Decoder(*DIMS, weights, 16, eager=eager)
    wait = lambda clocks, block: _ffi.check(_ffi.lib().nvllm_runner_step_wait(d.runner.h, clocks, block))
    d.sched.add_sequence(prompt, E.SamplingParams(temperature=0.0, max_tokens=len(forced), ignore_eos=True))
    got = []
    for i, t in enumerate(forced):
        b = d.sched.schedule()
        if i == 5:
            if where == "replay":
                d.runner.execute_model(b)
            wait(200000, silent)
            with pytest.raises(_ffi.NvllmError, match="in vain"):
                d.runner.execute_model(b) if where == "execute" else d.runner.replay_decode(2)
            wait(0, -1)
        got.append(d.runner.execute_model(b, return_logits=True)[1][0])
        if i == 6:
            assert d.runner.replay_decode(3) > 0
        d.sched.postprocess([int(t)])
    assert np.array_equal(np.stack(got), want)
