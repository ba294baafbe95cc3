"""The work a user of this framework has it do, as cases that can be timed and checked.

Families of cases, each through the public entry points of ``litnicelm_b200.plugin``:

* ``generate``   the token loop of the litnicelm transformer (``Session.generate``): greedy or sampled, one stream or
                 many in lockstep, the whole context recomputed per token or with cached keys and values. With the tokens
                 come the logits that follow the text, of sampled streams those that follow the prompts
                 (``Session.forward``).
* ``inspect``    the next-token distribution of whole prompts (``Session.inspect``).
* ``train``      one optimiser step of the transformer through the plugin table (``Backend``): forward, loss, backward,
                 clipping, AdamW, operator by operator as the host program issues them.
* ``prefill``    logits behind whole prompts of a registered design served from a model folder (``ModelSession.forward``).
* ``decode``     prompt and greedy continuation of a registered design (``ModelSession.generate``), and the logits that follow.
* ``extend``     one sequence fed in portions, logits of the wanted places (``ModelSession.extend``).

Models have the sizes of the repository's benchmark (widths 64, 512 and 1024, vocabularies of 8 to 32000) or sizes between
them, random weights, and for the registered designs a head that reads each token's successor off its embedding: as in a
trained model the most likely token leads clearly, so that rounding does not change a greedy continuation.
"""
import ctypes as C
import math
import os
import shutil
import tempfile

import numpy as np
import torch

from litnicelm_b200 import formats
from litnicelm_b200.plugin import Backend, DevTensor, ModelSession, Session


def _transformer(family, layers, heads, width, ff, vocab, max_seq, **more):
    return dict(family=family, layers=layers, heads=heads, width=width, ff=ff, vocab=vocab, max_seq=max_seq, **more)


def listed():
    char = dict(layers=6, heads=8, width=512, ff=2048, vocab=96, max_seq=1024)
    base = dict(heads=8, dim=64, width=512, ff=2048, vocab=8192)
    large = dict(heads=16, dim=64, width=1024, ff=4096, vocab=32000)
    return [
        # the smallest model of the benchmark, prompt and text of the smoke run: launches and latency
        _transformer("generate", 2, 2, 64, 256, 8, 64, name="generate-tiny", streams=1, prompt=6, new=58, sampled=False,
                     cached=False),
        # the headline: one stream of the character model, greedy, its context recomputed for every token
        dict(char, family="generate", name="generate-char", streams=1, prompt=256, new=256, sampled=False, cached=False),
        # the serving half of the headline: 64 streams in lockstep, sampled
        dict(char, family="generate", name="generate-char-64", streams=64, prompt=128, new=32, sampled=True, cached=False),
        # the same model with the cache option, as somebody runs it who wants the tokens soonest
        dict(char, family="generate", name="cached-char", streams=1, prompt=256, new=256, sampled=False, cached=True),
        dict(char, family="generate", name="cached-char-64", streams=64, prompt=128, new=64, sampled=True, cached=True),
        # whole prompts through the large transformer, the full distribution back
        _transformer("inspect", 12, 16, 1024, 4096, 32000, 2048, name="inspect-large", streams=8, prompt=2048),
        # a training step on the character model's layers, a batch of texts of no round length
        _transformer("train", 2, 8, 512, 2048, 96, 256, name="train-char", streams=8, prompt=250),
        # registered designs in bfloat16: prompts, one of them of no round length
        dict(large, family="prefill", name="mitilix-prefill", design="mitilix", dtype="bfloat16", layers=6, streams=4,
             prompt=2048),
        dict(large, family="prefill", name="gobesun-prefill", design="gobesun", dtype="bfloat16", layers=6, streams=4,
             prompt=2047),
        # answers of a few and of many streams
        dict(large, family="decode", name="mitilix-decode-8", design="mitilix", dtype="bfloat16", layers=12, streams=8,
             prompt=256, new=96),
        dict(base, family="decode", name="gobesun-decode-64", design="gobesun", dtype="bfloat16", layers=6, streams=64,
             prompt=200, new=96),
        # 32-bit arithmetic, a conversation fed in turns of very unequal lengths
        dict(base, family="extend", name="gobesun-extend-f32", design="gobesun", dtype="float32", layers=6, parts="613 1 1 37 300 1 9 1"),
    ]


def _between(rng, lo, hi):
    """A whole number, its logarithm evenly spread."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    family = rng.choice(["generate", "generate", "inspect", "train", "prefill", "decode", "extend"])
    if family in ("generate", "inspect", "train"):
        heads = rng.choice([2, 4, 8] if family != "inspect" else [4, 8, 16])
        width = heads * rng.choice([32, 64, 64])
        c = _transformer(family, rng.randint(1, 6), heads, width, width * rng.choice([2, 4]), _between(rng, 8, 1024), 1024)
        if family == "inspect":
            c.update(streams=_between(rng, 1, 8), prompt=_between(rng, 16, 1024), vocab=_between(rng, 96, 32000))
        elif family == "train":
            c.update(layers=rng.randint(1, 2), streams=_between(rng, 1, 8), prompt=_between(rng, 8, 256), max_seq=256)
        else:
            c.update(streams=_between(rng, 1, 64), sampled=rng.random() < 0.4, cached=rng.random() < 0.5)
            c["prompt"] = _between(rng, 4, 256)
            c["new"] = _between(rng, 8, 256 if c["streams"] <= 8 else 48)
        return c
    dim = rng.choice([32, 64])
    heads = rng.choice([4, 8, 16])
    width = max(256, heads * 64)
    c = dict(family=family, design=rng.choice(["mitilix", "gobesun"]), dtype="bfloat16", layers=rng.randint(3, 9), heads=heads,
             dim=dim, width=width, ff=width * rng.choice([2, 4]), vocab=_between(rng, 500, 16000))
    if family == "prefill":
        c.update(streams=_between(rng, 1, 8), prompt=_between(rng, 32, 2048))
    elif family == "decode":
        c.update(streams=_between(rng, 1, 64), prompt=_between(rng, 8, 256), new=_between(rng, 16, 96))
    else:
        parts = [_between(rng, 2, 600)] + [rng.choice([1, 1, _between(rng, 2, 300)]) for _ in range(rng.randint(3, 8))]
        c.update(dtype=rng.choice(["bfloat16", "float32"]), parts=" ".join(map(str, parts)))
    return c


# ---- weights and inputs ----------------------------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _dims(c):
    return formats.ModelDims(c["layers"], c["heads"], c["width"], c["ff"], c["vocab"], c["max_seq"])


def _arena(c, seed):
    """Parameter image: matrices N(0, 0.02), gains around one, shifts around zero. A model that generates has a head eight times
    that, as decided as a trained one (few near-equal candidates per draw); one in training has its hidden units clear of the
    ReLU's kink, where rounding would decide whether a unit has a gradient."""
    layout = formats.ParamLayout.build(_dims(c))
    values = torch.randn(layout.total_bytes // 4, generator=_generator(seed), device="cuda") * 0.02
    for name, (at, shape) in layout.slices.items():
        part = values[at // 4:at // 4 + shape[0] * shape[1]]
        if name.endswith("gamma"):
            part += 1.0
        elif name == "lm_head_w" and c["family"] == "generate":
            part *= 8.0
        elif name.endswith("ffn_b1") and c["family"] == "train":
            part[::2] += 3.0
            part[1::2] -= 3.0
    return layout, values


def _zipf(c, seed, count, length):
    return np.stack([formats.zipf_prompt(c["vocab"], length, 1000 * seed + i) for i in range(count)])


def _config(c):
    n, dim = c["layers"], c["dim"]
    if c["design"] == "mitilix":  # every third layer shares the latents before it
        layers = [{"heads": c["heads"], "dim": dim, "vdim": dim, "kv_rank": c["width"] // 4, "window": max(512, c["width"]),
                   "scale": dim ** -0.5, "ff": c["ff"], "kv_from": i - 1 if i % 3 == 2 else None} for i in range(n)]
        return formats.mitilix_config(c["width"], c["vocab"], 4096, layers, taps=4, eps=1e-6)
    layers, ff, own = [], (c["ff"] * 2 // 3 + 63) // 64 * 64, n * 2 // 3  # a third of the runs repeats
    for i in range(own):
        if i % 4 == 3:
            rot = {"dims": dim, "base": 5e5, "scaling": {"factor": 8.0, "original": 4096, "fast": 24.0, "slow": 2.0}}
            layers.append(formats.chunk_attention_layer(c["heads"], max(1, c["heads"] // 4), dim, dim, 2048, rot, ff=ff))
        else:
            d = 128 if c["width"] > 512 else 64
            layers.append(formats.delta_layer(c["width"] // d, c["width"] // d // 2, d, d, 4, ff=ff))
    return formats.gobesun_config(c["width"], c["vocab"], layers, (own - (n - own), own, 2), c["width"] ** 0.5, 1e-6)


def _successor(vocab):
    step = next(s for s in range(vocab // 3 + 1, 2 * vocab + 3) if math.gcd(s, vocab) == 1)
    return (np.arange(vocab) * step + 1) % vocab


def _design_weights(c, seed):
    """bfloat16 weights of a registered design on the device."""
    config, g = _config(c), _generator(seed)
    gobesun = c["design"] == "gobesun"
    out = {}
    for name, shape in (formats.gobesun_shapes if gobesun else formats.mitilix_shapes)(config).items():
        last = name.rsplit(".", 1)[-1]
        noise = torch.randn(shape, generator=g, device="cuda")
        if name == "embed":
            t = noise * (2.0 / (config["embedding"]["scale"] if gobesun else 1.0))
        elif name == "head":
            t = torch.empty_like(noise)
            t[torch.from_numpy(_successor(c["vocab"])).cuda()] = out["embed"].float() / out["embed"].float().square().sum(1).mean().sqrt()
        elif name == "pos":
            t = 0.3 * noise
        elif gobesun and (last in ("norm1", "norm1b", "norm2", "norm2b") or name == "final.norm"):
            t = 0.1 * noise
        elif last in ("norm", "norm1"):
            t = 1.0 + 0.1 * noise
        elif last == "A_log":
            t = torch.linspace(-4.0, 1.0, shape[0], device="cuda")
        elif last == "dt_bias":
            t = 0.5 * noise
        else:
            t = noise * shape[-1] ** -0.5
        out[name] = t.to(torch.bfloat16)
    return config, out


class _State:
    """Everything a case holds; its session is closed with it."""

    def __init__(self, **values):
        self.__dict__.update(values)

    def __del__(self):
        if getattr(self, "session", None) is not None:
            self.session.close()


def prepare(case, seed):
    c, family = dict(case), case["family"]
    if family == "train":
        return _prepare_training(c, seed)
    if family in ("generate", "inspect"):
        _, values = _arena(c, seed)
        cached = {"LITNICE_B200_KV_CACHE": "1"} if c.get("cached") else {}
        before = {k: os.environ.get(k) for k in cached}
        os.environ.update(cached)
        try:
            session = Session(_dims(c), c["streams"])
        finally:
            for k, v in before.items():
                os.environ.pop(k) if v is None else os.environ.update({k: v})
        state = _State(case=c, session=session, prompts=_zipf(c, seed, c["streams"], c["prompt"]),
                       seeds=np.arange(c["streams"], dtype=np.uint32) + np.uint32(seed % (1 << 31)))
        session.load_params(values.cpu().numpy().view(np.uint8))
        return state
    config, weights = _design_weights(c, seed)
    folder = tempfile.mkdtemp(prefix="model_")
    try:
        formats.write_model_folder(folder, config, {k: v.view(torch.int16).cpu().numpy().view(np.uint16) for k, v in weights.items()})
        session = ModelSession(folder, c["dtype"], c.get("streams", 1))
    finally:
        shutil.rmtree(folder, ignore_errors=True)
    rng = np.random.default_rng(seed)
    if family == "extend":
        tokens = [rng.integers(0, c["vocab"], int(n)).astype(np.int32) for n in c["parts"].split()]
        return _State(case=c, session=session, parts=tokens)
    return _State(case=c, session=session, prompts=rng.integers(0, c["vocab"], (c["streams"], c["prompt"])).astype(np.int32))


SAMPLING = dict(temp=0.8, top_k=40, top_p=0.95)


def run(state):
    c, s = state.case, getattr(state, "session", None)
    if c["family"] == "train":
        return _run_training(state)
    if c["family"] == "inspect":
        return s.inspect(state.prompts)
    if c["family"] == "prefill":
        return s.forward(state.prompts)
    if c["family"] == "extend":
        s.release(0)
        # the logits of the last place of every part, of the first part those of its middle too
        return [s.extend(0, p, [len(p) // 2, len(p) - 1] if i == 0 else [len(p) - 1]) for i, p in enumerate(state.parts)]
    if c.get("sampled"):  # which of two equal candidates is drawn changes a text: the logits are the prompts'
        return {"logits": s.forward(state.prompts), "tokens": s.generate(state.prompts, c["new"], seeds=state.seeds, **SAMPLING)}
    tokens = s.generate(state.prompts, c["new"])
    return {"tokens": tokens, "logits": s.forward(np.concatenate([state.prompts, tokens], 1)[:, -s.dims.max_seq:])}


# ---- a training step through the plugin table ------------------------------------------------------------------------

class _Plugin(Backend):
    """A plugin instance that lives as long as anybody holds it: the state, or a tensor on its memory."""

    def __del__(self):
        self.close()


class _DeviceFloats:
    def __init__(self, plugin, ptr, count):
        self.plugin = plugin
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f4", "data": (ptr, False), "version": 3}


LEARNING = dict(lr=3e-4, beta1=0.9, beta2=0.95, decay=0.1, clip=1.0)


def _prepare_training(c, seed):
    """The arenas of a model in training, and the operators of one step as (entry, arguments), their views made once."""
    be = _Plugin()
    layout, values = _arena(c, seed)
    total = layout.total_bytes
    B, S, D, F, V, H = c["streams"], c["prompt"], c["width"], c["ff"], c["vocab"], c["heads"]
    dh = D // H
    arena = {k: be.alloc(total) for k in ("params", "grads", "m", "v")}
    be.upload(arena["params"], values.cpu().numpy())
    for k in ("m", "v"):
        be.upload(arena[k], np.zeros(total, np.uint8))
    text = _zipf(c, seed, B, S + 1)
    keep = []

    def view(ptr, shape, strides=None, dtype=0):
        if strides is None:
            strides = [4 * int(np.prod(shape[i + 1:])) for i in range(len(shape))]
        v = DevTensor(ptr, tuple(shape), tuple(strides), dtype, be.device).view()
        keep.append(v)
        return C.byref(v)

    def buffer(*shape):
        return be.alloc(4 * int(np.prod(shape)))

    def dense(*shape):
        return view(buffer(*shape), shape)

    def p(name, which="params"):
        at, shape = layout.slices[name]
        return view(arena[which] + at, shape)

    def g(name):
        return p(name, "grads")

    ids, targets = be.alloc(4 * B * S), be.alloc(4 * B * S)
    be.upload(ids, np.ascontiguousarray(text[:, :-1]))
    be.upload(targets, np.ascontiguousarray(text[:, 1:]))
    ids, targets = view(ids, (B, S), dtype=1), view(targets, (B, S), dtype=1)
    ops = []

    def op(name, *args):
        ops.append((getattr(be.api, name), args))

    def projection(x, name, out):
        op("gemm_ranked_matrix_rhs", x, p(name + "_w"), out)
        op("add_bias_rowwise", out, p(name + "_b"), out)

    op("fill", view(arena["grads"], (1, total // 4)), 0.0)
    x = dense(B, S, D)
    at, shape = layout.slices["pos_embedding"]
    op("embedding_lookup", p("tok_embedding"), ids, x)
    op("add", x, view(arena["params"] + at, (S, D)), x)
    saved = []
    scale = float(np.float32(1.0) / np.sqrt(np.float32(dh)))
    for l in range(c["layers"]):
        n = f"layer{l}."
        k = dict(x=x, ln1=dense(B, S, D), qkv=buffer(B, S, 3 * D), weights=buffer(B, H, S, S), ctx=buffer(B, S, D), x1=dense(B, S, D),
                 ln2=dense(B, S, D), h=dense(B, S, F))
        saved.append(k)
        out, x = dense(B, S, D), dense(B, S, D)
        op("layernorm_forward", k["x"], p(n + "ln1_gamma"), p(n + "ln1_beta"), k["ln1"])
        projection(k["ln1"], n + "attn_qkv", view(k["qkv"], (B, S, 3 * D)))
        third = lambda ptr, i, h: view(ptr + 4 * (i * D + h * dh), (B, S, dh), (12 * S * D, 12 * D, 4))  # noqa: E731
        head = lambda ptr, h: view(ptr + 4 * h * dh, (B, S, dh), (4 * S * D, 4 * D, 4))  # noqa: E731
        square = lambda ptr, h: view(ptr + 4 * h * S * S, (B, S, S), (4 * H * S * S, 4 * S, 4))  # noqa: E731
        k.update(third=third, head=head, square=square)
        for h in range(H):
            w = square(k["weights"], h)
            op("gemm_batched_rhs_t", third(k["qkv"], 0, h), third(k["qkv"], 1, h), w)
            op("scaled_causal_softmax_rows", w, scale, w)
            op("gemm_batched", w, third(k["qkv"], 2, h), head(k["ctx"], h))
        projection(view(k["ctx"], (B, S, D)), n + "attn_out", out)
        op("add", k["x"], out, k["x1"])
        op("layernorm_forward", k["x1"], p(n + "ln2_gamma"), p(n + "ln2_beta"), k["ln2"])
        op("gemm_ranked_matrix_rhs", k["ln2"], p(n + "ffn_w1"), k["h"])
        op("add_bias_relu_rowwise_inplace", k["h"], p(n + "ffn_b1"))
        op("gemm_ranked_matrix_rhs", k["h"], p(n + "ffn_w2"), out)
        op("add_bias_rowwise", out, p(n + "ffn_b2"), out)
        op("add", k["x1"], out, x)
    last, logits, loss = dense(B, S, D), dense(B, S, V), dense(1, 1)
    op("layernorm_forward", x, p("lnf_gamma"), p("lnf_beta"), last)
    op("gemm_ranked_matrix_rhs", last, p("lm_head_w"), logits)
    op("cross_entropy_mean_backward_inplace", logits, targets, loss)
    dx, dn, dadd, dff, dctx, dqkv = dense(B, S, D), dense(B, S, D), dense(B, S, D), dense(B, S, F), buffer(B, S, D), buffer(B, S, 3 * D)
    dw = dense(B, S, S)
    op("gemm_ranked_reduce_lhs_t", last, logits, g("lm_head_w"))
    op("gemm_ranked_matrix_rhs_t", logits, p("lm_head_w"), dn)
    op("layernorm_backward", x, p("lnf_gamma"), dn, dx, g("lnf_gamma"), g("lnf_beta"))
    for l in reversed(range(c["layers"])):
        n, k = f"layer{l}.", saved[l]
        op("row_sum", dx, g(n + "ffn_b2"))
        op("gemm_ranked_reduce_lhs_t", k["h"], dx, g(n + "ffn_w2"))
        op("gemm_ranked_matrix_rhs_t", dx, p(n + "ffn_w2"), dff)
        op("relu_backward_inplace", k["h"], dff)
        op("row_sum", dff, g(n + "ffn_b1"))
        op("gemm_ranked_reduce_lhs_t", k["ln2"], dff, g(n + "ffn_w1"))
        op("gemm_ranked_matrix_rhs_t", dff, p(n + "ffn_w1"), dn)
        op("layernorm_backward", k["x1"], p(n + "ln2_gamma"), dn, dadd, g(n + "ln2_gamma"), g(n + "ln2_beta"))
        op("add_inplace", dx, dadd)
        op("row_sum", dx, g(n + "attn_out_b"))
        op("gemm_ranked_reduce_lhs_t", view(k["ctx"], (B, S, D)), dx, g(n + "attn_out_w"))
        op("gemm_ranked_matrix_rhs_t", dx, p(n + "attn_out_w"), view(dctx, (B, S, D)))
        for h in range(H):
            w, third = k["square"](k["weights"], h), k["third"]
            op("gemm_batched_lhs_t", w, k["head"](dctx, h), third(dqkv, 2, h))
            op("gemm_batched_rhs_t", k["head"](dctx, h), third(k["qkv"], 2, h), dw)
            op("softmax_backward_causal_rows", w, dw, dw)
            op("mul_scalar", dw, scale, dw)
            op("gemm_batched", dw, third(k["qkv"], 1, h), third(dqkv, 0, h))
            op("gemm_batched_lhs_t", dw, third(k["qkv"], 0, h), third(dqkv, 1, h))
        whole = view(dqkv, (B, S, 3 * D))
        op("row_sum", whole, g(n + "attn_qkv_b"))
        op("gemm_ranked_reduce_lhs_t", k["ln1"], whole, g(n + "attn_qkv_w"))
        op("gemm_ranked_matrix_rhs_t", whole, p(n + "attn_qkv_w"), dn)
        op("layernorm_backward", k["x"], p(n + "ln1_gamma"), dn, dadd, g(n + "ln1_gamma"), g(n + "ln1_beta"))
        op("add_inplace", dx, dadd)
    op("accumulate_embedding_grads", ids, dx, g("tok_embedding"), g("pos_embedding"))
    cut = layout.decay_bytes
    zones = [{k: view(a + at, (1, n // 4)) for k, a in arena.items()} for at, n in ((0, cut), (cut, total - cut))]
    return _State(case=c, backend=be, keep=keep, ops=ops, loss=loss, zones=zones, step=0, all_grads=view(arena["grads"], (1, total // 4)),
                  outputs={k: _DeviceFloats(be, a, total // 4) for k, a in arena.items()})


def _run_training(state):
    h, api, z = state.backend.h, state.backend.api, LEARNING
    for entry, args in state.ops:
        entry(h, *args)
    norm = math.sqrt(api.sum_squares_f32(h, state.all_grads))
    if norm > z["clip"]:
        api.mul_scalar(h, state.all_grads, z["clip"] / norm, state.all_grads)
    state.step += 1
    for i, zone in enumerate(state.zones):
        api.adamw_step(h, zone["params"], zone["grads"], zone["m"], zone["v"], state.step, z["lr"], z["beta1"], z["beta2"],
                       z["decay"], 1 if i == 0 else 0)
    loss = api.read_scalar_f32(h, state.loss)
    return {"loss": loss, **{k: torch.as_tensor(v, device="cuda") for k, v in state.outputs.items()}}


# ---- what a pass cannot do without -----------------------------------------------------------------------------------

def _design_sizes(c):
    """(weights the layer runs read, flops of mixing per token at a mean context n, bytes of state per token and stream)."""
    config = _config(c)
    if c["design"] == "mitilix":
        runs = config["layers"]
    else:
        lp, layers = config["loop"], config["layers"]
        runs = layers[:lp["start"]] + layers[lp["start"]:lp["stop"]] * lp["times"] + layers[lp["stop"]:]
    d, weights, fixed, per_key, window = c["width"], 0, 0.0, 0.0, 1 << 30
    for e in runs:
        m = e["mixer"]
        q, o = m["heads"] * m["dim"], m["heads"] * m["vdim"]
        weights += d * o + (3 if c["design"] == "gobesun" else 2) * d * e["mlp"]["ff"]
        if e["type"] == "latent_attention":
            weights += d * q + m["kv_rank"] * (q + o + (d if m.get("kv_from") is None else 0))
            per_key += 2.0 * (q + o)
            window = m["mask"]["size"]
        elif e["type"] == "delta":
            kv = m["kv_heads"] * m["dim"]
            weights += d * (2 * kv + 2 * o + 2 * m["heads"])
            fixed += 6.0 * o * m["dim"]
        else:
            weights += d * (q + m["kv_heads"] * (m["dim"] + m["vdim"]))
            per_key += 2.0 * (q + o)
    return weights, fixed, per_key, window


def work(case):
    c, f = dict(case), case["family"]
    if f in ("generate", "inspect", "train"):
        D, F, L, V, B, P = c["width"], c["ff"], c["layers"], c["vocab"], c["streams"], c["prompt"]
        matrices = L * (4 * D * D + 2 * D * F)
        forward = lambda s: 2.0 * s * matrices + 2.0 * L * s * (s + 1) * D + 2.0 * D * V  # noqa: E731
        if f == "inspect":
            return {"bytes": 4.0 * (matrices + D * V + B * V), "flops": B * forward(P)}
        if f == "train":
            rows = B * P
            return {"bytes": 4.0 * 7 * formats.ParamLayout.build(_dims(c)).total_bytes / 4,
                    "flops": 3.0 * (2.0 * rows * (matrices + D * V) + 2.0 * L * B * P * (P + 1) * D)}
        n = min(c["new"], c["max_seq"] - P)
        # every token reads every weight; the loop recomputes its context by contract unless keys and values are cached
        steps = [forward(P + i) for i in range(n)] if not c["cached"] else [forward(P)] + [
            2.0 * (matrices + D * V) + 4.0 * L * (P + i) * D for i in range(1, n)]
        cache = sum(8.0 * L * D * (P + i) for i in range(1, n)) * B if c["cached"] else 0.0
        extra = P if c["sampled"] else P + n
        return {"bytes": 4.0 * (n + 1) * (matrices + D * V) + cache, "flops": B * (sum(steps) + forward(extra))}
    weights, fixed, per_key, window = _design_sizes(c)
    head, es = c["width"] * c["vocab"], 2.0 if c["dtype"] == "bfloat16" else 4.0

    def rows(a, b):  # positions a .. b - 1 of one sequence
        return (b - a) * (2.0 * weights + fixed) + per_key * sum(min(i + 1, window) for i in range(a, b))

    if f == "prefill":
        return {"bytes": es * (weights + head) + 4.0 * c["streams"] * c["vocab"], "flops": c["streams"] * (rows(0, c["prompt"]) + 2.0 * head)}
    if f == "decode":
        end = c["prompt"] + c["new"]
        return {"bytes": es * (weights + head) * (c["new"] + 1),
                "flops": c["streams"] * (rows(0, end - 1) + rows(0, end) + 2.0 * head * (c["new"] + 1))}
    parts = [int(n) for n in c["parts"].split()]
    return {"bytes": es * (weights + head) * len(parts), "flops": rows(0, sum(parts)) + 2.0 * head * (len(parts) + 1)}


def tolerance(case):
    """About four times the errors against 64 bits that were measured: 1e-7 to 5e-6 in 32 bits, 0.003 to 0.009 in bfloat16."""
    if case["family"] == "inspect":
        return {"rel": 1e-5}
    if case["family"] == "train":
        return {"rel": 1e-5, "max": 0.1}  # AdamW's first steps divide gradients by their own size: tiny ones may change sign
    if case["family"] == "generate":
        return {"rel": 1e-5, "differ": 0.01}  # ties, draws beside an edge
    if case["dtype"] == "float32":
        return {"rel": 2e-5}
    return {"rel": 0.015 if case["design"] == "mitilix" else 0.03, "differ": 0.01}


# ---- the same in 64 bits, plain torch ----------------------------------------------------------------------------------

def _layernorm(x, g, b):
    return torch.nn.functional.layer_norm(x, x.shape[-1:], g.reshape(-1), b.reshape(-1), float(np.float32(1e-5)))


def _causal(q, k, v, scale, seen):
    w = (q @ k.transpose(-1, -2) * scale).masked_fill(~seen, -math.inf)
    return torch.softmax(w, -1) @ v


def _transformer_logits(c, p, ids, last_only=True):
    B, S = ids.shape
    D, H = c["width"], c["heads"]
    x = p["tok_embedding"][ids] + p["pos_embedding"][:S]
    seen = torch.ones(S, S, dtype=torch.bool, device="cuda").tril()
    for l in range(c["layers"]):
        n = f"layer{l}."
        h = _layernorm(x, p[n + "ln1_gamma"], p[n + "ln1_beta"]) @ p[n + "attn_qkv_w"] + p[n + "attn_qkv_b"]
        q, k, v = (t.reshape(B, S, H, D // H).transpose(1, 2) for t in h.split(D, -1))
        o = _causal(q, k, v, (D // H) ** -0.5, seen).transpose(1, 2).reshape(B, S, D)
        x = x + o @ p[n + "attn_out_w"] + p[n + "attn_out_b"]
        h = _layernorm(x, p[n + "ln2_gamma"], p[n + "ln2_beta"])
        x = x + torch.relu(h @ p[n + "ffn_w1"] + p[n + "ffn_b1"]) @ p[n + "ffn_w2"] + p[n + "ffn_b2"]
    if last_only:
        x = x[:, -1]
    return _layernorm(x, p["lnf_gamma"], p["lnf_beta"]) @ p["lm_head_w"]


class _Draws:
    """std::mt19937 with std::discrete_distribution behind temperature, top-k and top-p."""

    def __init__(self, seed):
        self.words = np.random.RandomState(int(seed))

    def pick(self, logits):
        x = logits / float(np.float32(SAMPLING["temp"]))
        order = np.argsort(-x, kind="stable")[:SAMPLING["top_k"]]
        w = np.exp(x[order] - x[order[0]])
        p = np.cumsum(w) / w.sum()
        keep = min(len(p), int(np.searchsorted(p, float(np.float32(SAMPLING["top_p"])))) + 1)
        if keep < 2:
            return int(order[0])
        a, b = (int(v) for v in self.words.randint(0, 1 << 32, 2, dtype=np.uint32))
        edges = np.cumsum(w[:keep] / w[:keep].sum())
        edges[-1] = 1.0
        return int(order[np.searchsorted(edges, (a + b * 4294967296.0) / 18446744073709551616.0)])


def _continue(logits_of, prompts, new, sampled, seeds):
    """Prompts and their continuation. Greedy: guessed, and guessed again from the logits over all of it until nothing changes.
    logits_of(ids, last_only)."""
    B, P = prompts.shape
    ids = torch.from_numpy(prompts).long().cuda()
    if sampled:
        draws = [_Draws(s) for s in seeds]
        for _ in range(new):
            rows = logits_of(ids, True).cpu().numpy()
            ids = torch.cat([ids, torch.tensor([[d.pick(r)] for d, r in zip(draws, rows)], device="cuda")], 1)
        return ids
    ids = torch.cat([ids, torch.zeros(B, new, dtype=torch.long, device="cuda")], 1)
    for _ in range(new + 1):  # every pass settles one more token at least
        said = logits_of(ids, False)[:, P - 1:-1].argmax(-1)
        if bool((said == ids[:, P:]).all()):
            break
        ids[:, P:] = said
    return ids


def _rms(x, eps):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)


def _channel_conv(h, w):
    taps = w.shape[1]
    padded = torch.nn.functional.pad(h, (0, 0, taps - 1, 0))
    return sum(padded[:, j:j + h.shape[1]] * w[:, j] for j in range(taps))


def _mitilix(config, w, ids, last_only=False):
    B, T = ids.shape
    eps, latents = config["norm"]["eps"], {}
    x = w["embed"][ids] + w["pos"][:T]
    i, j = torch.arange(T, device="cuda")[:, None], torch.arange(T, device="cuda")[None]
    for n, e in enumerate(config["layers"]):
        m, p = e["mixer"], f"l{n}."
        h = _rms(x, eps) * w[p + "norm1"]
        a = h + _channel_conv(h, w[p + "canon1"])
        if m.get("kv_from") is None:
            latents[n] = _rms(a @ w[p + "mix.dkv"].T, eps) * w[p + "mix.dkv.norm"]
        c = latents[n if m.get("kv_from") is None else m["kv_from"]]
        heads = lambda t: t.reshape(B, T, m["heads"], -1).transpose(1, 2)  # noqa: E731
        seen = (i >= j) & (i - j < m["mask"]["size"])
        o = _causal(heads(a @ w[p + "mix.q"].T), heads(c @ w[p + "mix.uk"].T), heads(c @ w[p + "mix.uv"].T), m["scale"], seen)
        y = o.transpose(1, 2).reshape(B, T, -1) @ w[p + "mix.o"].T
        up = torch.nn.functional.gelu((h + _channel_conv(h, w[p + "canon2"])) @ w[p + "mlp.up"].T)
        x = x + y + up @ w[p + "mlp.down"].T
    if last_only:
        x = x[:, -1]
    return _rms(x, eps) * w["final.norm"] @ w["head"].T


def _turn(x, rot):
    dims, sc = rot["dims"], rot["scaling"]
    f = rot["base"] ** (-2.0 * np.arange(dims // 2) / dims)
    place = lambda turns: dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(rot["base"]))  # noqa: E731
    lo, hi = max(math.floor(place(sc["fast"])), 0), min(math.ceil(place(sc["slow"])), dims - 1)
    ramp = np.clip((np.arange(dims // 2) - lo) / max(hi - lo, 0.001), 0.0, 1.0)
    f = torch.from_numpy(f / sc["factor"] * ramp + f * (1.0 - ramp)).cuda()
    angle = (torch.arange(x.shape[1], device="cuda", dtype=torch.float64)[:, None] * f)[None, :, None]
    amplitude = 0.1 * math.log(sc["factor"]) + 1.0
    co, si = torch.cos(angle) * amplitude, torch.sin(angle) * amplitude
    u, v = x[..., :dims // 2], x[..., dims // 2:dims]
    return torch.cat([u * co - v * si, v * co + u * si, x[..., dims:]], -1)


def _gobesun(config, w, ids, last_only=False):
    B, T = ids.shape
    eps, lp = config["norm"]["eps"], config["loop"]
    x = w["embed"][ids] * config["embedding"]["scale"]
    order = list(range(lp["start"])) + list(range(lp["start"], lp["stop"])) * lp["times"] + list(range(lp["stop"], len(config["layers"])))
    at = torch.arange(T, device="cuda")
    for n in order:
        e, p = config["layers"][n], f"l{n}."
        m, t = e["mixer"], f"l{n}.mix."
        H, G, dim, vdim = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        h = _rms(x, eps) * (1.0 + w[p + "norm1"])
        if e["type"] == "delta":
            q, k, v = (torch.nn.functional.silu(_channel_conv(h @ w[t + s].T, w[t + s + ".conv"])) for s in "qkv")
            unit = lambda z: z / torch.sqrt(z.square().sum(-1, keepdim=True) + 1e-6)  # noqa: E731
            q, k = (unit(z.reshape(B, T, G, dim)).repeat_interleave(H // G, 2) for z in (q, k))
            q, v = q * dim ** -0.5, v.reshape(B, T, H, vdim)
            beta = torch.sigmoid(h @ w[t + "b"].T)
            decay = torch.exp(-torch.exp(w[t + "A_log"]) * torch.nn.functional.softplus(h @ w[t + "a"].T + w[t + "dt_bias"]))
            s, o = torch.zeros(B, H, dim, vdim, dtype=x.dtype, device="cuda"), torch.empty_like(v)
            for i in range(T):
                s *= decay[:, i, :, None, None]
                u = beta[:, i, :, None] * (v[:, i] - (k[:, i, :, None] @ s)[:, :, 0])
                s += k[:, i, :, :, None] * u[:, :, None]
                o[:, i] = (q[:, i, :, None] @ s)[:, :, 0]
            o = _rms(o, eps) * w[t + "norm"] * torch.nn.functional.silu(h @ w[t + "g"].T).reshape(B, T, H, vdim)
        else:
            q = (_rms(h @ w[t + "q"].T, eps) * w[t + "q.norm"]).reshape(B, T, H, dim)
            k = (_rms(h @ w[t + "k"].T, eps) * w[t + "k.norm"]).reshape(B, T, G, dim)
            v = (h @ w[t + "v"].T).reshape(B, T, G, vdim)
            q, k = _turn(q, m["rot"]), _turn(k, m["rot"])
            k, v = (z.repeat_interleave(H // G, 2).transpose(1, 2) for z in (k, v))
            size = m["mask"]["size"]
            seen = (at[:, None] >= at[None]) & (at[:, None] // size == at[None] // size)
            o = _causal(q.transpose(1, 2), k, v, m["scale"], seen).transpose(1, 2)
        x = x + _rms(o.reshape(B, T, -1) @ w[t + "o"].T, eps) * (1.0 + w[p + "norm1b"])
        h = _rms(x, eps) * (1.0 + w[p + "norm2"])
        f = torch.nn.functional.gelu(h @ w[p + "mlp.gate"].T, approximate="tanh") * (h @ w[p + "mlp.up"].T)
        x = x + _rms(f @ w[p + "mlp.down"].T, eps) * (1.0 + w[p + "norm2b"])
    if last_only:
        x = x[:, -1]
    return (_rms(x, eps) * (1.0 + w["final.norm"])) @ w["head"].T


def _exact_training(c, layout, p, seed):
    text = torch.from_numpy(_zipf(c, seed, c["streams"], c["prompt"] + 1)).long().cuda()
    with torch.enable_grad():
        p = {k: v.requires_grad_() for k, v in p.items()}
        logits = _transformer_logits(c, p, text[:, :-1], last_only=False)
        loss = torch.nn.functional.cross_entropy(logits.reshape(-1, c["vocab"]), text[:, 1:].reshape(-1))
        loss.backward()
    z, flat = LEARNING, {}
    norm = math.sqrt(sum(float(v.grad.square().sum()) for v in p.values()))
    shrink = z["clip"] / norm if norm > z["clip"] else 1.0
    for k in ("params", "grads", "m", "v"):
        flat[k] = torch.zeros(layout.total_bytes // 4, dtype=torch.float64, device="cuda")
    b1, b2, lr, decay = (float(np.float32(z[k])) for k in ("beta1", "beta2", "lr", "decay"))
    for name, (at, shape) in layout.slices.items():
        v, gr = p[name].detach(), p[name].grad * shrink
        m, s = (1.0 - b1) * gr, (1.0 - b2) * gr * gr
        step = (m / (1.0 - b1)) / (torch.sqrt(s / (1.0 - b2)) + 1e-8) + (decay * v if at < layout.decay_bytes else 0.0)
        for k, t in (("params", v - lr * step), ("grads", gr), ("m", m), ("v", s)):
            flat[k][at // 4:at // 4 + shape[0] * shape[1]] = t.reshape(-1)
    if layout.total_bytes != sum(4 * s[0] * s[1] for _, s in layout.slices.values()):
        flat["params"] = None  # alignment gaps hold values of their own
    return {"loss": float(loss), **flat}


@torch.no_grad()
def exact(case, seed):
    c, f = dict(case), case["family"]
    if f in ("generate", "inspect", "train"):
        layout, values = _arena(c, seed)
        p = {k: values[at // 4:at // 4 + s[0] * s[1]].reshape(s).double() for k, (at, s) in layout.slices.items()}
        if f == "train":
            return _exact_training(c, layout, p, seed)
        prompts = _zipf(c, seed, c["streams"], c["prompt"])
        if f == "inspect":
            rows = [_transformer_logits(c, p, torch.from_numpy(prompts[i:i + 1]).long().cuda()) for i in range(len(prompts))]
            return torch.softmax(torch.cat(rows), -1)
        new = min(c["new"], c["max_seq"] - c["prompt"])
        seeds = np.arange(c["streams"], dtype=np.uint32) + np.uint32(seed % (1 << 31))
        ids = _continue(lambda i, last: _transformer_logits(c, p, i, last), prompts, new, c["sampled"], seeds)
        behind = ids[:, :c["prompt"]] if c["sampled"] else ids[:, -c["max_seq"]:]
        return {"tokens": ids[:, c["prompt"]:].int(), "logits": _transformer_logits(c, p, behind)}
    config, w = _design_weights(c, seed)
    w = {k: v.double() for k, v in w.items()}
    model = _mitilix if c["design"] == "mitilix" else _gobesun
    rng = np.random.default_rng(seed)
    if f == "extend":
        parts = [rng.integers(0, c["vocab"], int(n)) for n in c["parts"].split()]
        rows = model(config, w, torch.from_numpy(np.concatenate(parts)).cuda()[None])[0]
        ends = np.cumsum([len(t) for t in parts])
        return [rows[[len(parts[0]) // 2, ends[0] - 1] if i == 0 else [n - 1]] for i, n in enumerate(ends)]
    prompts = rng.integers(0, c["vocab"], (c["streams"], c["prompt"])).astype(np.int32)
    if f == "prefill":
        return model(config, w, torch.from_numpy(prompts).long().cuda(), True)
    after, ids = _successor(c["vocab"]), prompts
    for _ in range(c["new"]):  # the head reads successors: a guess that one pass confirms
        ids = np.concatenate([ids, after[ids[:, -1:]].astype(np.int32)], 1)
    ids = torch.from_numpy(ids).long().cuda()
    logits = torch.cat([model(config, w, ids[i:i + 16])[:, c["prompt"] - 1:] for i in range(0, len(ids), 16)])
    if not bool((logits[:, :-1].argmax(-1) == ids[:, c["prompt"]:]).all()):
        return None
    return {"tokens": ids[:, c["prompt"]:].int(), "logits": logits[:, -1]}
