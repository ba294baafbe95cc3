"""Projections of many rows (resident CTAs over 128 x 256 tiles) against the oracle: row counts that are no multiple of a
tile, the last tile of a wave, graph replay with fewer rows than the launch was sized for, and the pass that fills the caches."""
import numpy as np
import pytest

from litnicelm_b200 import formats
from litnicelm_b200.plugin import Session

pytestmark = pytest.mark.gpu


# (layers, heads, width, ff), streams, prompt, new: thirds of 256 columns and thirds that share a tile, one and several
# waves of tiles
@pytest.mark.parametrize("dims,streams,prompt,new", [
    ((2, 4, 256, 512), 64, 60, 7),
    ((1, 8, 512, 1024), 47, 126, 4),
    ((1, 4, 256, 256), 150, 90, 3),
    ((2, 12, 768, 768), 31, 129, 3),
])
@pytest.mark.parametrize("cached", [False, True])
def test_many_rows_against_the_oracle(oracle, monkeypatch, dims, streams, prompt, new, cached):
    if cached:
        monkeypatch.setenv("LITNICE_B200_KV_CACHE", "1")
    d = formats.ModelDims(*dims, 96, 160)
    arena = formats.make_param_arena(d, 11, bias_std=0.02, ln_std=0.1)
    prompts = np.stack([formats.zipf_prompt(d.vocab, prompt, 40 + i) for i in range(streams)])
    with Session(d, streams) as s:
        s.load_params(arena)
        whole = s.forward(prompts)
        fast = s.generate(prompts, new)          # graph replay: launches sized for the bucket's bound
        s.keep_step_logits(True)
        toks = s.generate(prompts, new)
        lg = s.read_step_logits(new, streams)
    for b in sorted({0, 1, streams // 2, streams - 1}):
        ref_tokens, ref_logits = oracle.generate(d, arena, prompts[b], new, want_logits=True)
        scale = np.abs(ref_logits).max(-1, keepdims=True)
        srt = np.sort(ref_logits.astype(np.float64), axis=1)
        ties = np.flatnonzero((toks[b] != ref_tokens) | (fast[b] != ref_tokens))
        n = int(ties[0]) if len(ties) else new
        assert n == new or srt[n, -1] - srt[n, -2] < 1e-4
        # operands of 22 bits (2^-22 per product), sums of at most 1024 terms in fp32 on either side, two layers
        assert float((np.abs(lg[:n, b] - ref_logits[:n]) / scale[:n]).max()) < 2e-5
        assert float((np.abs(whole[b] - ref_logits[0]) / scale[0]).max()) < 2e-5
