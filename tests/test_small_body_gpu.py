"""All layers of a small model in one launch against the oracle: row counts around a block of eight and a cluster's share, every
head dimension, several streams, contexts that grow through a graph's bucket and past what the launch is used for."""
import numpy as np
import pytest

from litnicelm_b200 import formats
from litnicelm_b200.plugin import Session

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,streams,prompt,new", [
    ((2, 2, 64, 256, 8, 64), 1, 1, 63),
    ((1, 4, 64, 100, 33, 130), 3, 57, 20),
    ((3, 1, 16, 48, 11, 90), 2, 63, 9),
    ((2, 2, 32, 32, 20, 40), 5, 8, 9),
    ((1, 2, 128, 512, 96, 100), 2, 59, 9),
    ((2, 3, 96, 384, 40, 80), 1, 31, 6),
    ((1, 1, 128, 256, 30, 64), 2, 17, 4),
])
def test_small_models_against_the_oracle(oracle, dims, streams, prompt, new):
    d = formats.ModelDims(*dims)
    arena = formats.make_param_arena(d, 5, bias_std=0.02, ln_std=0.1)
    prompts = np.stack([formats.zipf_prompt(d.vocab, prompt, 90 + i) for i in range(streams)])
    with Session(d, streams) as s:
        s.load_params(arena)
        every = s.forward(prompts, all_rows=True)
        fast = s.generate(prompts, new)
        s.keep_step_logits(True)
        toks = s.generate(prompts, new)
        lg = s.read_step_logits(new, streams)
    for b in range(streams):
        ref_tokens, ref_logits = oracle.generate(d, arena, prompts[b], new, want_logits=True)
        scale = np.abs(ref_logits).max(-1, keepdims=True)
        srt = np.sort(ref_logits.astype(np.float64), axis=1)
        ties = np.flatnonzero((toks[b] != ref_tokens) | (fast[b] != ref_tokens))
        n = int(ties[0]) if len(ties) else new
        assert n == new or srt[n, -1] - srt[n, -2] < 1e-4
        # sums of at most 512 terms in fp32 on either side (2^-24 each step, in different orders), three layers
        assert float((np.abs(lg[:n, b] - ref_logits[:n]) / scale[:n]).max()) < 2e-5
        whole = oracle.forward(d, arena, prompts[b])
        assert float((np.abs(every[b] - whole) / np.abs(whole).max()).max()) < 2e-5


def test_bad_ids_are_errors():
    d = formats.ModelDims(1, 2, 64, 128, 9, 32)
    with Session(d, 1) as s:
        s.load_params(formats.make_param_arena(d, 5))
        with pytest.raises(Exception, match="id out of range"):
            s.forward(np.array([[1, 2, 9]], np.int32))
