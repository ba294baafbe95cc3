"""All layers of a small model in one launch against the oracle: row counts around a block of eight and a cluster's share, every
head dimension, several streams, contexts that grow through a graph's bucket and past what the launch is used for."""
import os

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


# Greedy runs in one launch: vocabularies of any size up to what shared memory holds of the head, then token by token; texts that
# start shorter than the cluster's share; one layer and three (the two buffers change roles from step to step); runs resumed.
@pytest.mark.parametrize("dims,streams,prompt,new", [
    ((1, 2, 64, 128, 1, 40), 1, 2, 30),
    ((3, 2, 64, 256, 37, 70), 4, 6, 60),
    ((1, 2, 32, 64, 300, 128), 15, 60, 60),
    ((2, 2, 64, 256, 400, 60), 2, 20, 30),
    ((2, 4, 128, 256, 130, 64), 1, 1, 62),
])
def test_runs_in_one_launch(oracle, dims, streams, prompt, new):
    d = formats.ModelDims(*dims)
    arena = formats.make_param_arena(d, 5, bias_std=0.02, ln_std=0.1)
    prompts = np.stack([formats.zipf_prompt(d.vocab, prompt, 90 + i) for i in range(streams)])
    with Session(d, streams) as s:
        s.load_params(arena)
        whole = s.generate(prompts, new)
        s.upload_prompts(prompts)
        assert s.run(new // 3) == new // 3 and s.run(new - new // 3) == new
        parts = s.download_tokens(new)
        s.keep_step_logits(True)
        toks = s.generate(prompts, new)
        lg = s.read_step_logits(new, streams)
    assert np.array_equal(whole, parts)
    for b in range(streams):
        ties = np.flatnonzero(whole[b] != toks[b])
        if len(ties):
            srt = np.sort(lg[ties[0], b].astype(np.float64))
            assert srt[-1] - srt[-2] < 1e-4
    ref_tokens, ref_logits = oracle.generate(d, arena, prompts[-1], new, want_logits=True)
    srt = np.sort(ref_logits.astype(np.float64), axis=1)
    ties = np.flatnonzero(whole[-1] != ref_tokens)
    assert not len(ties) or srt[ties[0], -1] - srt[ties[0], -2] < 1e-4


def test_bad_ids_are_errors():
    d = formats.ModelDims(1, 2, 64, 128, 9, 32)
    with Session(d, 1) as s:
        s.load_params(formats.make_param_arena(d, 5))
        with pytest.raises(Exception, match="id out of range"):
            s.forward(np.array([[1, 2, 9]], np.int32))


@pytest.mark.parametrize("width,heads", [(32, 2), (64, 2), (96, 3)])
def test_rows_far_from_zero(oracle, width, heads):
    """Embeddings a million away from zero, half apart: the first LayerNorm's variance comes out of such rows as the host's two
    passes give it. What it feeds is scaled up so that the stream's own rounding (1/16 at a million) does not count."""
    d = formats.ModelDims(1, heads, width, 2 * width, 20, 48)
    arena = formats.make_param_arena(d, 5)
    layout = formats.ParamLayout.build(d)
    rng = np.random.default_rng(width)
    layout.view(arena, "tok_embedding")[...] = 1.0e6 + np.round(4.0 * rng.standard_normal((20, width))) / 8.0
    layout.view(arena, "pos_embedding")[...] = 0.0
    layout.view(arena, "layer0.attn_out_w")[...] *= 1e8
    layout.view(arena, "layer0.ffn_w2")[...] *= 1e4
    ids = rng.integers(0, 20, (2, 19)).astype(np.int32)
    with Session(d, 2) as s:
        s.load_params(arena)
        got = s.forward(ids, all_rows=True)
    for b in range(2):
        want = oracle.forward(d, arena, ids[b])
        assert float(np.abs(got[b] - want).max() / np.abs(want).max()) < 2e-5


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("place", [0, 37])
def test_values_that_are_not_finite_stay_visible(oracle, value, place):
    """One of them in a token's embedding: the logits of its row and of those behind it are not numbers, as the host's are."""
    d = formats.ModelDims(2, 2, 64, 128, 20, 48)
    arena = formats.make_param_arena(d, 5)
    formats.ParamLayout.build(d).view(arena, "tok_embedding")[3, place] = value
    ids = np.array([1, 2, 4, 5, 3, 6, 7, 8, 9, 10, 11], np.int32)
    with Session(d, 1) as s:
        s.load_params(arena)
        got = s.forward(ids, all_rows=True)[0]
    assert np.isnan(oracle.forward(d, arena, ids)[4:]).all() and np.isnan(got[4:]).all()
    before = oracle.forward(d, arena, ids[:4])
    assert float(np.abs(got[:4] - before).max() / np.abs(before).max()) < 2e-5


def test_profile_of_the_path_that_runs():
    """profile_step times what the token loop launches: all layers at once, or operator by operator where that is asked for."""
    d = formats.ModelDims(2, 2, 64, 256, 8, 64)
    stats = {}
    for small in ("1", "0"):
        os.environ["LITNICE_B200_SMALL"] = small
        try:
            with Session(d, 2) as s:
                s.load_params(formats.make_param_arena(d, 5))
                stats[small] = s.profile_step(2, 40, 3)
        finally:
            del os.environ["LITNICE_B200_SMALL"]
    head = stats["0"].gemm_launches - 3 * 2 * 4  # of the operators' run, beside four projections per layer
    assert stats["0"].attn_launches == 3 * 2 and stats["1"].attn_launches == 0
    assert stats["1"].gemm_launches == 3 + head and stats["1"].gemm_flops == stats["0"].gemm_flops
    assert 0 < stats["1"].gemm_ms < stats["0"].gemm_ms + stats["0"].attn_ms
