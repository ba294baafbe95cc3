"""Calls that a host makes head by head (attention, forward and backward) are recorded and issued over all heads at once where
that writes the same values: every buffer of a run must hold the same bits as when each call is issued at once."""
import os

import numpy as np
import pytest
import torch

from litnicelm_b200.plugin import Backend, DevTensor

pytestmark = pytest.mark.gpu

B, S, H, DH = 2, 24, 4, 16   # below the extents of the tensor-core products: sums in the order of k on either route
D = H * DH


class Arena:
    """Buffers of one instance, filled alike in every instance."""

    def __init__(self, be):
        self.be, self.buffers = be, {}

    def buffer(self, name, floats):
        rng = np.random.default_rng(sum(map(ord, name)))
        values = (rng.standard_normal(floats) * 0.5).astype(np.float32)
        ptr = self.be.alloc(values.nbytes, 64)
        self.be.upload(ptr, values.view(np.uint8))
        self.buffers[name] = (ptr, values.nbytes)
        return ptr

    def read(self):
        return {k: self.be.download(p, n) for k, (p, n) in self.buffers.items()}


def view(ptr, shape, strides=None):
    if strides is None:
        strides = [4 * int(np.prod(shape[i + 1:])) for i in range(len(shape))]
    return DevTensor(ptr, tuple(shape), tuple(strides), 0, 1)


def third(ptr, i, h):
    return view(ptr + 4 * (i * D + h * DH), (B, S, DH), (12 * S * D, 12 * D, 4))


def head(ptr, h):
    return view(ptr + 4 * h * DH, (B, S, DH), (4 * S * D, 4 * D, 4))


def square(ptr, h):
    return view(ptr + 4 * h * S * S, (B, S, S), (4 * H * S * S, 4 * S, 4))


def forward(be, a, shared, scale=0.25):
    qkv, w, ctx, tmp = a.buffer("qkv", 3 * B * S * D), a.buffer("w", B * H * S * S), a.buffer("ctx", B * S * D), a.buffer("tmp", B * S * S)
    for h in range(H):
        s = view(tmp, (B, S, S)) if shared else square(w, h)
        be.call("gemm_batched_rhs_t", third(qkv, 0, h), third(qkv, 1, h), s)
        be.call("scaled_causal_softmax_rows", s, scale, square(w, h))
        be.call("gemm_batched", square(w, h), third(qkv, 2, h), head(ctx, h))


def backward(be, a, variant):
    qkv, w, dctx = a.buffer("qkv", 3 * B * S * D), a.buffer("w", B * H * S * S), a.buffer("dctx", B * S * D)
    dqkv, tmp, more = a.buffer("dqkv", 3 * B * S * D), a.buffer("tmp", B * S * S), a.buffer("more", B * H * S * S)
    for h in range(H):
        dw = square(more, h) if variant == "own" else view(tmp, (B, S, S))
        scale = 0.25 + 0.125 * h if variant == "scales" else {"negative scale": -0.25, "infinite scale": np.inf}.get(variant, 0.25)
        dv = third(dqkv, 2, 0 if variant == "one gradient" else h)
        k = third(qkv, 1, h)
        if variant == "next head reads":   # a head's key is what the head before it wrote
            k = third(dqkv, 0, max(h - 1, 0))
        be.call("gemm_batched_lhs_t", square(w, h), head(dctx, h), dv)
        if variant == "not filled":        # what the shared buffer holds is used before a head fills it
            be.call("mul_scalar", dw, 0.5, dw)
            be.call("gemm_batched", dw, third(qkv, 0, h), third(dqkv, 1, h))
        if variant == "exec":
            be.call("gemm_batched_rhs_t_exec_context", head(dctx, h), third(qkv, 2, h), dw)
            be.call("softmax_backward_causal_rows_exec_context", square(w, h), dw, dw)
        else:
            be.call("gemm_batched_rhs_t", head(dctx, h), third(qkv, 2, h), dw)
            be.call("softmax_backward_causal_rows", square(w, h), dw, dw)
        if variant == "last incomplete" and h == H - 1:
            break
        if variant != "not scaled":
            be.call("mul_scalar", dw, scale, dw)
        if variant == "other view":        # the shared buffer through another view of itself
            be.call("gemm_batched", view(tmp, (B, S, S), (4 * S * S, 4, 4 * S)), k, third(dqkv, 0, h))
        else:
            be.call("gemm_batched", dw, k, third(dqkv, 0, h))
        be.call("gemm_batched_lhs_t", dw, third(qkv, 0, h), third(dqkv, 1, h))


def uneven(be, a):
    """Two heads of the usual pitch and one somewhere else."""
    x, y = a.buffer("x", 4 * S * S), a.buffer("y", 8 * S * S)
    for at in (0, 1, 3):
        v = view(x + 4 * at * S * S, (1, S, S))
        be.call("gemm_batched_rhs_t", v, v, view(y + 4 * (at if at < 2 else 7) * S * S, (1, S, S)))


def running(be, a):
    """Each product reads what the one before it wrote."""
    x = a.buffer("x", 6 * S * S)
    for at in range(5):
        v = view(x + 4 * at * S * S, (1, S, S))
        be.call("gemm_batched_rhs_t", v, v, view(x + 4 * (at + 1) * S * S, (1, S, S)))


def overlapping(be, a):
    """Results half over their neighbours'."""
    x, y = a.buffer("x", 4 * S * S), a.buffer("y", 4 * S * S)
    for at in range(4):
        v = view(x + 4 * at * S * S, (1, S, S))
        be.call("gemm_batched_lhs_t", v, v, view(y + 2 * at * S * S, (1, S, S)))


def backwards(be, a):
    """Addresses that fall from head to head."""
    x, y = a.buffer("x", 4 * S * S), a.buffer("y", 4 * S * S)
    for at in (3, 2, 1, 0):
        v = view(x + 4 * at * S * S, (1, S, S))
        be.call("gemm_batched_lhs_t", v, v, view(y + 4 * at * S * S, (1, S, S)))


def vectors(be, a, op):
    """Row calls on views of rank 1 between the products."""
    x, y, z = a.buffer("x", H * S * S), a.buffer("y", H * S * S), a.buffer("z", 3 * H * S)
    for h in range(H):
        m, out = view(x + 4 * h * S * S, (1, S, S)), view(y + 4 * h * S * S, (1, S, S))
        u, v, w = (view(z + 4 * (i * H + h) * S, (S,)) for i in range(3))
        be.call("gemm_batched_lhs_t", m, m, out)
        if op == "mul_scalar":
            be.call(op, u, 0.5, v)
        elif op == "scaled_causal_softmax_rows":
            be.call(op, u, 0.5, v)
        else:
            be.call(op, u, v, w)


def one_right_operand(be, a, op):
    """A head's batch shares its right operand, which has no batch axis, or one of extent 1."""
    x, y, z = a.buffer("x", H * B * S * S), a.buffer("y", H * S * S), a.buffer("z", H * B * S * S)
    for h in range(H):
        shape = (S, S) if op == "gemm_batched_rhs_t" else (1, S, S)
        be.call(op, view(x + 4 * h * B * S * S, (B, S, S)), view(y + 4 * h * S * S, shape), view(z + 4 * h * B * S * S, (B, S, S)))


def small_products(be, a):
    """More products of 2 x 2 than a grid has layers, each call alone within them."""
    batch = 20000
    x, y = a.buffer("x", H * batch * 4), a.buffer("y", H * batch * 4)
    for h in range(H):
        m = view(x + 16 * h * batch, (batch, 2, 2))
        be.call("gemm_batched_rhs_t", m, m, view(y + 16 * h * batch, (batch, 2, 2)))


def lanes(be, a):
    be.call("start_exec_context_iteration")
    be.call("start_exec_context_group")
    backward(be, a, "exec")
    be.call("finish_exec_context_group")
    be.call("finish_exec_context_iteration")


RUNS = {"forward": lambda be, a: forward(be, a, False), "forward, one score buffer": lambda be, a: forward(be, a, True),
        "uneven": uneven, "running": running, "small products": small_products, "overlapping": overlapping, "backwards": backwards, "exec": lanes}
for name in ("shared", "own", "scales", "one gradient", "next head reads", "not filled", "not scaled", "other view", "last incomplete", "negative scale",
             "infinite scale"):
    RUNS["backward, " + name] = lambda be, a, name=name: backward(be, a, name)
GROUPED = {"small products", "forward", "forward, one score buffer", "exec", "backward, shared", "backward, own", "backward, not scaled",
           "backward, last incomplete", "backward, negative scale", "backward, infinite scale"}


def rectangular(be, a, rows, cols, batch):
    """A causal row's limit is its number among the rows of its call, modulo the columns: heads whose rows are no whole squares."""
    def mat(name, h, m, n):
        return view(a.buffers[name][0] + 4 * h * batch * m * n, (batch, m, n))
    for name, floats in (("q", rows * DH), ("k", cols * DH), ("w", rows * cols), ("ctx", rows * DH), ("dw", rows * cols), ("dq", rows * DH)):
        a.buffer(name, H * batch * floats)
    for h in range(H):
        w = mat("w", h, rows, cols)
        be.call("gemm_batched_rhs_t", mat("q", h, rows, DH), mat("k", h, cols, DH), w)
        be.call("scaled_causal_softmax_rows", w, 0.25, w)
        be.call("gemm_batched", w, mat("k", h, cols, DH), mat("ctx", h, rows, DH))
    be.download(*a.buffers["q"])         # (a run ends at any other call)
    for h in range(H):
        dw = mat("dw", h, rows, cols)
        be.call("gemm_batched_rhs_t", mat("ctx", h, rows, DH), mat("k", h, cols, DH), dw)
        be.call("softmax_backward_causal_rows", mat("w", h, rows, cols), dw, dw)
        be.call("gemm_batched", dw, mat("k", h, cols, DH), mat("dq", h, rows, DH))


for rows, cols, batch in ((24, 32, 1), (32, 24, 1), (24, 32, 2), (3, 5, 1), (48, 24, 1), (24, 48, 2)):
    name = f"causal {batch} x {rows} x {cols}"
    RUNS[name] = lambda be, a, size=(rows, cols, batch): rectangular(be, a, *size)
    if batch * rows % cols == 0:
        GROUPED.add(name)


for op in ("mul_scalar", "scaled_causal_softmax_rows", "softmax_backward_causal_rows"):
    RUNS[op + " of vectors"] = lambda be, a, op=op: vectors(be, a, op)
GROUPED.add("mul_scalar of vectors")


for op in ("gemm_batched_rhs_t", "gemm_batched_lhs_t"):
    RUNS[op + ", one right operand"] = lambda be, a, op=op: one_right_operand(be, a, op)


@pytest.mark.parametrize("name", RUNS)
def test_same_bits_as_call_by_call(name):
    left, launches = [], []
    for queue in ("1", "0"):
        os.environ["LITNICE_B200_ABI_QUEUE"] = queue
        try:
            be = Backend()
        finally:
            del os.environ["LITNICE_B200_ABI_QUEUE"]
        with be:
            a = Arena(be)
            with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
                RUNS[name](be, a)
                left.append(a.read())
            launches.append(sum("kernel" in e.name for e in prof.events()))
    for k in left[0]:
        assert np.array_equal(left[0][k], left[1][k]), k
    assert (launches[0] < launches[1]) == (name in GROUPED), launches


def test_long_sums_stay_on_the_tensor_cores():
    """Heads whose operands in parts pass the 4 GB up to which a product has room for them, each alone far below: no head may go
    to the plain tiles for the others' sake. Blocks of 64 k are added with rounding, in ranges that need not be the same: errors of
    2^-24 that add up like a walk."""
    heads, k = 32, 163840
    left = []
    for queue in ("1", "0"):
        os.environ["LITNICE_B200_ABI_QUEUE"] = queue
        try:
            be = Backend()
        finally:
            del os.environ["LITNICE_B200_ABI_QUEUE"]
        with be:
            a = Arena(be)
            x, y = a.buffer("x", (heads + 64) * k), a.buffer("y", heads * 64 * 64)
            with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
                for h in range(heads):
                    m = view(x + 4 * h * k, (1, 64, k))
                    be.call("gemm_batched_rhs_t", m, m, view(y + 4 * h * 64 * 64, (1, 64, 64)))
                left.append(be.download(*a.buffers["y"]).view(np.float32))
            names = {e.name for e in prof.events()}
            assert any("gemm_split" in n for n in names) and not any("gemm_simt" in n for n in names), names
    assert np.linalg.norm(left[0] - left[1]) < 2 ** -24 * (k / 64) ** 0.5 * np.linalg.norm(left[0])


def test_kept_memory_is_given_back():
    """What the calls of heads keep (here 256 MB) does not stand in the way of the host's own allocations."""
    heads, n = 8, 2048 * 4
    with Backend() as be:
        x, y = be.alloc(heads * n * 2 * 4, 64), be.alloc(n * n // 8 * 4, 64)
        be.call("fill", view(x, (heads * n * 2,)), 1.0)
        out = view(y, (1, n // 8, n))
        for h in range(heads):
            be.call("gemm_batched_rhs_t", view(x + 8 * n * h, (1, n // 8, 2)), view(x + 8 * n * h, (1, n, 2)), out)
        be.download(y, 4)
        whole = be.api.memory_info(be.h).free_bytes + (128 << 20)
        be.api.free(be.h, be.api.alloc(be.h, whole, 64))
