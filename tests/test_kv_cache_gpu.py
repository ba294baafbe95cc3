"""The opt-in cached mode (LITNICE_B200_KV_CACHE=1) against the oracle.

The reference keeps no key/value cache: every token recomputes its whole
context (inference.cpp:278-284). The cached mode is an extension that must
not change results: same logits within 1e-3 of the row's largest magnitude,
same greedy tokens except at logged near-ties (top-2 gap < 1e-4), same sampled
tokens, the loop guard of inference.cpp:278, resumed runs, several streams.
"""
import hashlib
import os

import numpy as np
import pytest
import torch

from litnicelm_b200 import formats
from litnicelm_b200.plugin import Session
from conftest import GOLDEN, load_small

pytestmark = pytest.mark.gpu

LOGIT_RTOL = 1e-3
NEAR_TIE = 1e-4


def rel_err(got, want):
    scale = np.maximum(np.abs(want).max(axis=-1, keepdims=True), 1e-6)
    return float((np.abs(got - want) / scale).max())


@pytest.fixture(autouse=True)
def cached_mode():
    old = os.environ.get("LITNICE_B200_KV_CACHE")
    os.environ["LITNICE_B200_KV_CACHE"] = "1"
    yield
    if old is None:
        del os.environ["LITNICE_B200_KV_CACHE"]
    else:
        os.environ["LITNICE_B200_KV_CACHE"] = old


def agreed_prefix(tokens, ref_tokens, gaps):
    assert len(tokens) == len(ref_tokens)
    for i, (a, b) in enumerate(zip(tokens, ref_tokens)):
        if a != b:
            assert gaps[i] < NEAR_TIE, f"step {i}: token {a} != {b} with top-2 gap {gaps[i]}"
            print(f"near-tie at step {i}: gap {gaps[i]:.3e}; comparison stops here")
            return i
    return len(tokens)


@pytest.mark.parametrize("name", ["c1", "abcdef"])
def test_small_models_tokens_and_step_logits(name):
    d, z = load_small(name)
    srt = np.sort(z["greedy_step_logits"].astype(np.float64), axis=1)
    gaps = srt[:, -1] - srt[:, -2]
    with Session(d, 4) as s:
        s.load_params(z["arena"])
        s.keep_step_logits(True)
        toks = s.generate(z["prompt"], 128)[0]
        lg = s.read_step_logits(len(toks), 1)[:, 0, :]
        s.keep_step_logits(False)
        fast = s.generate(z["prompt"], 128)[0]      # graph replay
        temp, top_k, top_p, seed = z["sampled_params"]
        sampled = s.generate(z["prompt"], 128, temp=float(temp), top_k=int(top_k), top_p=float(top_p),
                             seeds=[int(seed)])[0]
    n = agreed_prefix(toks, z["greedy_tokens"], gaps)
    assert rel_err(lg[:n], z["greedy_step_logits"][:n]) < LOGIT_RTOL
    assert np.array_equal(fast, toks)
    assert len(toks) == min(128, d.max_seq - len(z["prompt"]))   # loop guard of inference.cpp:278
    agree = int(np.argmin(np.append(sampled == z["sampled_tokens"], False)))
    assert agree >= min(len(z["sampled_tokens"]), 8)


def test_config2_bench_workload_in_cached_mode():
    z = np.load(os.path.join(GOLDEN, "c2_full.npz"))
    d = formats.CONFIG_DIMS["c2"]
    arena = formats.make_param_arena(d, int(z["arena_seed"][0]))
    if hashlib.sha256(arena.tobytes()).digest() != z["arena_sha256"].tobytes():
        pytest.skip("numpy's generator stream changed; the seeded arena no longer matches the fixture")
    with Session(d, 1) as s:
        s.load_params(arena)
        fast = s.generate(z["prompt"], 768)[0]
        s.keep_step_logits(True)
        toks = s.generate(z["prompt"], 768)[0]
        lg = s.read_step_logits(len(toks), 1)[:, 0, :]
    n = agreed_prefix(toks, z["greedy_tokens"], z["top2_gap"])
    err = rel_err(lg[:n], z["logits_all"][255:255 + n])
    print(f"cached mode, config 2: {n}/768 tokens identical, step logits {err:.2e}")
    assert err < LOGIT_RTOL
    agreed_prefix(fast, z["greedy_tokens"], z["top2_gap"])


def test_streams_resume_and_many_streams(oracle):
    d = formats.ModelDims(2, 4, 128, 256, 50, 96)
    arena = formats.make_param_arena(d, 99, bias_std=0.02, ln_std=0.1)
    prompts = np.stack([formats.zipf_prompt(d.vocab, 17, 500 + i) for i in range(12)])
    ref = [oracle.generate(d, arena, p, 20, want_logits=True) for p in prompts]
    with Session(d, 12) as s:
        s.load_params(arena)
        few = s.generate(prompts[:3], 20)              # few-row products
        many = s.generate(prompts, 20)                 # more than 8 streams: tile kernel
        s.upload_prompts(prompts[:3])
        assert s.run(7) == 7
        assert s.run(13) == 20                         # resumes on the caches
        parts = s.download_tokens(20)
        s.keep_step_logits(True)
        s.generate(prompts[:3], 20)
        lg = s.read_step_logits(20, 3)
    for b in range(12):
        srt = np.sort(ref[b][1].astype(np.float64), axis=1)
        agreed_prefix(many[b], ref[b][0], srt[:, -1] - srt[:, -2])
        if b < 3:
            agreed_prefix(few[b], ref[b][0], srt[:, -1] - srt[:, -2])
    assert np.array_equal(parts, few)
    for b in range(3):
        assert rel_err(lg[:, b, :], ref[b][1]) < LOGIT_RTOL


# More than 8 streams: steps on the tensor cores. Every head dimension (64: fp16 pairs, others: TF32 pairs), one and several
# key chunks, contexts that cross a 64-position bucket, heads on the tensor cores (vocabulary % 64 == 0), in the one-launch
# tail, and on the tile kernel.
@pytest.mark.parametrize("dims,streams,prompt,new", [
    ((2, 2, 128, 256, 64, 160), 9, 60, 20),
    ((1, 3, 192, 192, 50, 300), 33, 40, 12),
    ((2, 4, 128, 256, 52, 96), 12, 1, 9),
    ((1, 1, 128, 128, 96, 200), 9, 130, 10),
    ((1, 8, 128, 192, 128, 80), 129, 62, 6),
])
def test_many_streams_step_on_the_tensor_cores(oracle, dims, streams, prompt, new):
    d = formats.ModelDims(*dims)
    arena = formats.make_param_arena(d, 7, bias_std=0.02, ln_std=0.1)
    prompts = np.stack([formats.zipf_prompt(d.vocab, prompt, 70 + i) for i in range(streams)])
    with Session(d, streams) as s:
        s.load_params(arena)
        fast = s.generate(prompts, new)
        s.keep_step_logits(True)
        toks = s.generate(prompts, new)
        lg = s.read_step_logits(new, streams)
    for b in sorted({0, 7, 8, streams // 2, streams - 1}):
        ref_tokens, ref_logits = oracle.generate(d, arena, prompts[b], new, want_logits=True)
        srt = np.sort(ref_logits.astype(np.float64), axis=1)
        gaps = srt[:, -1] - srt[:, -2]
        n = agreed_prefix(toks[b], ref_tokens, gaps)
        # operands of 22 bits (2^-22 per product), sums of at most 256 terms in fp32 on either side, a handful of layers
        assert rel_err(lg[:n, b, :], ref_logits[:n]) < 2e-5
        agreed_prefix(fast[b], ref_tokens, gaps)


# Steps launched one by one (their logits are kept) see contexts between the multiples of 64 that a replayed step is sized for:
# 48 heads cut 193 .. 224 positions into more chunks than any multiple up to 256, 16 heads 577 .. 608.
@pytest.mark.parametrize("dims,streams,prompt,new", [
    ((2, 2, 64, 128, 24, 300), 24, 200, 24),
    ((1, 2, 128, 128, 30, 640), 8, 590, 20),
])
def test_contexts_between_the_buckets(oracle, dims, streams, prompt, new):
    d = formats.ModelDims(*dims)
    arena = formats.make_param_arena(d, 7, bias_std=0.02, ln_std=0.1)
    prompts = np.stack([formats.zipf_prompt(d.vocab, prompt, 70 + i) for i in range(streams)])
    with Session(d, streams) as s:
        s.load_params(arena)
        fast = s.generate(prompts, new)
        s.keep_step_logits(True)
        toks = s.generate(prompts, new)
        lg = s.read_step_logits(new, streams)
    for b in range(streams):
        ref_tokens, ref_logits = oracle.generate(d, arena, prompts[b], new, want_logits=True)
        srt = np.sort(ref_logits.astype(np.float64), axis=1)
        gaps = srt[:, -1] - srt[:, -2]
        n = agreed_prefix(toks[b], ref_tokens, gaps)
        assert rel_err(lg[:n, b, :], ref_logits[:n]) < 2e-5  # as above
        agreed_prefix(fast[b], ref_tokens, gaps)


def logits_64(d, arena, ids):
    """Logits [rows, vocab] of one text in 64 bits."""
    p = {k: formats.ParamLayout.build(d).view(arena, k).astype(np.float64) for k in formats.ParamLayout.build(d).slices}

    def norm(x, name):
        m = x.mean(-1, keepdims=True)
        return (x - m) / np.sqrt(((x - m) ** 2).mean(-1, keepdims=True) + np.float32(1e-5)) * p[name + "_gamma"] + p[name + "_beta"]

    x = p["tok_embedding"][ids] + p["pos_embedding"][:len(ids)]
    dh = d.d_model // d.n_heads
    for l in range(d.n_layers):
        n = f"layer{l}."
        h = norm(x, n + "ln1") @ p[n + "attn_qkv_w"] + p[n + "attn_qkv_b"]
        q, k, v = (t.reshape(len(ids), d.n_heads, dh).transpose(1, 0, 2) for t in np.split(h, 3, -1))
        s = np.where(np.tri(len(ids), dtype=bool), q @ k.transpose(0, 2, 1) / np.sqrt(dh), -np.inf)
        w = np.exp(s - s.max(-1, keepdims=True))
        o = (w / w.sum(-1, keepdims=True)) @ v
        x = x + o.transpose(1, 0, 2).reshape(len(ids), -1) @ p[n + "attn_out_w"] + p[n + "attn_out_b"]
        h = norm(x, n + "ln2")
        x = x + np.maximum(h @ p[n + "ffn_w1"] + p[n + "ffn_b1"], 0.0) @ p[n + "ffn_w2"] + p[n + "ffn_b2"]
    return norm(x, "lnf") @ p["lm_head_w"]


@pytest.mark.parametrize("dims,streams,prompt,new", [
    ((2, 4, 256, 512, 40, 200), 12, 70, 6),     # steps and prompt on fp16 pairs
    ((2, 8, 256, 1024, 96, 120), 40, 20, 6),    # head dimension 32: TF32 pairs
    ((1, 8, 512, 2048, 96, 300), 9, 200, 4),
    ((2, 4, 256, 1024, 30, 300), 2, 230, 12),   # the prompt alone
    ((2, 2, 64, 256, 24, 300), 7, 200, 12),     # narrow, few streams: 32-bit throughout
])
def test_error_not_above_the_32_bit_kernels(dims, streams, prompt, new):
    """Step logits against 64 bits, in the 2-norm: where operands are split in two 16- or 19-bit parts, no further off than the
    same run on the fp32 kernels."""
    d = formats.ModelDims(*dims)
    arena = formats.make_param_arena(d, 7, bias_std=0.02, ln_std=0.1)
    prompts = np.stack([formats.zipf_prompt(d.vocab, prompt, 70 + i) for i in range(streams)])
    off = []
    for tc in ("1", "0"):
        os.environ["LITNICE_B200_TC"] = tc
        try:
            with Session(d, streams) as s:
                s.load_params(arena)
                s.keep_step_logits(True)
                toks = s.generate(prompts, new)
                lg = s.read_step_logits(new, streams)
        finally:
            del os.environ["LITNICE_B200_TC"]
        total = 0.0
        for b in sorted({0, streams // 2, streams - 1}):
            want = logits_64(d, arena, np.concatenate([prompts[b], toks[b][:-1]]))[prompt - 1:]
            total += ((lg[:, b] - want) ** 2).sum() / (want ** 2).sum()
        off.append(total)
    assert off[0] <= off[1]


# Greedy steps in one resident kernel: a cluster per head (1, 2, 4 or 8 heads of 32 or 64), else a CTA per SM (three heads).
# Every number of streams its rows are compiled for and those between; contexts of one and several batches of keys per warp,
# shorter than the cluster; one and several passes of every product, vocabularies of one column, with a remainder, of several
# tiles per CTA; hidden widths at both ends of what a cluster takes.
@pytest.mark.parametrize("dims,streams,prompt,new", [
    ((2, 2, 64, 256, 8, 64), 1, 3, 60),
    ((1, 1, 32, 32, 1, 40), 1, 1, 12),
    ((2, 1, 64, 1024, 33, 90), 3, 5, 30),
    ((2, 2, 128, 64, 51, 330), 8, 300, 25),
    ((3, 4, 128, 512, 1000, 200), 5, 130, 40),
    ((2, 4, 256, 512, 96, 1300), 1, 1240, 30),
    ((2, 8, 256, 1024, 7, 260), 2, 200, 50),
    ((2, 8, 512, 2048, 96, 400), 1, 250, 40),
    ((1, 8, 512, 2048, 9000, 300), 4, 60, 12),
    ((2, 8, 512, 1024, 130, 160), 7, 100, 24),
    ((2, 3, 96, 256, 52, 120), 2, 40, 20),
])
def test_resident_steps(dims, streams, prompt, new):
    d = formats.ModelDims(*dims)
    arena = formats.make_param_arena(d, 7, bias_std=0.02, ln_std=0.1)
    prompts = np.stack([formats.zipf_prompt(d.vocab, prompt, 70 + i) for i in range(streams)])
    with Session(d, streams) as s:
        s.load_params(arena)
        whole = s.generate(prompts, new)
        s.upload_prompts(prompts)
        first = new // 2
        assert s.run(first) == first
        s.keep_step_logits(True)
        assert s.run(new - first) == new  # launched one by one, on the keys and values that the resident kernel left
        toks = s.download_tokens(new)
        lg = s.read_step_logits(new, streams)[first:]
    # sums of up to 1024 terms in fp32 on either side: as in the tests above
    for b in range(streams):
        for run in (whole, toks):
            want = logits_64(d, arena, np.concatenate([prompts[b], run[b][:-1]]))[prompt - 1:]
            srt = np.sort(want, axis=1)
            gaps = srt[:, -1] - srt[:, -2] if d.vocab > 1 else np.ones(new)
            agreed_prefix(run[b], want.argmax(1), gaps)
        assert rel_err(lg[:, b], want[first:]) < 2e-5
    if streams > 1:  # a stream's tokens do not depend on its neighbours
        with Session(d, streams) as s:
            s.load_params(arena)
            alone = s.generate(prompts[1:2], new)[0]
        want = logits_64(d, arena, np.concatenate([prompts[1], alone[:-1]]))[prompt - 1:]
        srt = np.sort(want, axis=1)
        agreed_prefix(alone, want.argmax(1), srt[:, -1] - srt[:, -2])


def test_only_greedy_runs_hold_the_resident_kernels_weights():
    """The kernel's copy of the weights (44 MB here) is made for the first run that uses it."""
    d = formats.ModelDims(1, 8, 512, 2048, 16000, 64)
    prompts = np.stack([formats.zipf_prompt(d.vocab, 20, 70 + i) for i in range(2)])
    free = []
    with Session(d, 2) as s:
        s.load_params(formats.make_param_arena(d, 7, bias_std=0.02, ln_std=0.1))
        for more in (dict(temp=0.8, top_k=20, seeds=[1, 2]), dict()):
            for _ in range(2):
                s.generate(prompts, 8, **more)
            free.append(torch.cuda.mem_get_info()[0])
    assert 40 << 20 < free[0] - free[1] < 64 << 20


# Up to 64 rows a step on the weights' pairs: tiles of rows that are not full, one, two and four of them a CTA, one span of k for a
# part of the warps, for all of them and several; past 64 rows and past width 512 the tiles of the large products.
@pytest.mark.parametrize("dims,streams,prompt,new", [
    ((2, 1, 64, 64, 30, 60), 9, 20, 5),
    ((2, 3, 192, 576, 50, 60), 23, 30, 4),
    ((2, 8, 512, 2048, 96, 70), 64, 40, 4),
    ((1, 8, 512, 512, 40, 70), 41, 20, 4),
    ((1, 4, 256, 1024, 40, 70), 65, 20, 3),
    ((1, 10, 640, 1280, 40, 60), 12, 20, 3),
])
def test_steps_of_tens_of_rows(dims, streams, prompt, new):
    d = formats.ModelDims(*dims)
    arena = formats.make_param_arena(d, 7, bias_std=0.02, ln_std=0.1)
    prompts = np.stack([formats.zipf_prompt(d.vocab, prompt, 70 + i) for i in range(streams)])
    with Session(d, streams) as s:
        s.load_params(arena)
        fast = s.generate(prompts, new)
        s.keep_step_logits(True)
        toks = s.generate(prompts, new)
        lg = s.read_step_logits(new, streams)
    for b in sorted({0, 7, 8, streams // 2, streams - 1}):
        want = logits_64(d, arena, np.concatenate([prompts[b], toks[b][:-1]]))[prompt - 1:]
        # operands of 22 bits, sums of at most 2048 terms in fp32: as above
        assert rel_err(lg[:, b], want) < 2e-5
        same = np.flatnonzero(fast[b] != toks[b])
        srt = np.sort(want, axis=1)
        assert not len(same) or srt[same[0], -1] - srt[same[0], -2] < NEAR_TIE


# The step's attention by batches of keys a warp: one that is not full, one that is, several with the next on its way, several without
# (more CTAs than are resident with it); heads of 32, 64 and 128; chunks joined, and one that writes its context by itself.
@pytest.mark.parametrize("dims,streams,prompt,new", [
    ((1, 16, 512, 128, 24, 150), 64, 62, 5),
    ((1, 16, 512, 128, 24, 150), 64, 124, 5),
    ((1, 16, 1024, 128, 24, 60), 64, 31, 4),
    ((1, 16, 1024, 128, 24, 80), 48, 62, 5),
    ((1, 8, 1024, 128, 24, 100), 9, 14, 5),
    ((1, 8, 1024, 128, 24, 100), 60, 70, 5),
    ((1, 4, 128, 128, 24, 700), 12, 640, 5),
])
def test_attention_of_a_step_by_batches(dims, streams, prompt, new):
    test_steps_of_tens_of_rows(dims, streams, prompt, new)
