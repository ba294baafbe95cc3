"""The plugin table's products at sizes that run on the tensor cores, against 64-bit sums: tile edges and remainders, strides
of every kind, summed and batched operands, cut k ranges, epilogues, values that no operand parts hold, and what the parts keep of those they hold."""
import time

import numpy as np
import pytest

from abi_util import Buffer
from litnicelm_b200 import formats
from litnicelm_b200.plugin import Backend, ModelSession
from mitilix_util import layer
from training_util import dense, read, sliced

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    b = Backend()
    yield b
    b.close()


def operand(be, a, layout):
    """`a` in a buffer of its own as rows of k, turned, or with gaps that no 16-byte access fits."""
    if layout == "rows":
        return dense(be, a)[1]
    turned = np.swapaxes(a, -1, -2)
    if layout == "turned":
        t = dense(be, np.ascontiguousarray(turned))[1]
        s = list(t.strides)
        return type(t)(t.ptr, a.shape, tuple(s[:-2] + [s[-1], s[-2]]), t.dtype, t.device)
    pitch = a.shape[-1] + 3
    wide = np.full(a.shape[:-1] + (pitch,), -7.0, np.float32)
    wide[..., 1:1 + a.shape[-1]] = a
    t = dense(be, wide)[1]
    return type(t)(t.ptr + 4, a.shape, t.strides, t.dtype, t.device)


def bound(a, b):
    """What the operands' parts leave out is below 2^-32 of a product; a chain of 64 k loses up to 2^-23 of its sum at each of four
    truncations, every chain 2^-24 at each of two roundings: below 2^-21 |a| |b| in all. Short sums run one after another in 32 bits:
    2^-24 a step."""
    k = a.shape[-1]
    return max(2.0 ** -21, k * 2.0 ** -24 if k < 128 else 0.0) * (np.abs(a.astype(np.float64)) @ np.abs(b.astype(np.float64))) + 1e-30


@pytest.mark.parametrize("m,n,k", [(128, 128, 1024), (129, 130, 1030), (1, 500, 5000), (300, 64, 900), (2000, 96, 512),
                                   (127, 2050, 260), (1500, 1290, 72), (640, 3000, 33), (24, 40, 4096)])
@pytest.mark.parametrize("left,right", [("rows", "rows"), ("turned", "gaps"), ("gaps", "turned")])
def test_product(be, m, n, k, left, right):
    rng = np.random.default_rng(m + n + k)
    a = (rng.standard_normal((m, k)) * 10.0 ** rng.uniform(-6, 6, (m, 1))).astype(np.float32)
    b = (rng.standard_normal((k, n)) * 10.0 ** rng.uniform(-6, 6, (1, n))).astype(np.float32)
    ob, ov = dense(be, np.zeros((m, n), np.float32))
    be.call("gemm", operand(be, a, left), operand(be, b, right), ov)
    want = a.astype(np.float64) @ b.astype(np.float64)
    assert (np.abs(read(ob, ov) - want) <= bound(a, b)).all()


@pytest.mark.parametrize("batch,m,n,k", [(8, 250, 250, 64), (3, 130, 70, 513), (64, 100, 64, 100), (2, 300, 700, 96)])
def test_batches_sums_and_epilogues(be, batch, m, n, k):
    rng = np.random.default_rng(batch + m + n + k)
    a = rng.standard_normal((batch, m, k)).astype(np.float32)
    b = rng.standard_normal((batch, k, n)).astype(np.float32)
    ob, ov = dense(be, np.zeros((batch, m, n), np.float32))
    be.call("gemm_batched", operand(be, a, "gaps"), operand(be, b, "rows"), ov)
    want = a.astype(np.float64) @ b.astype(np.float64)
    assert (np.abs(read(ob, ov) - want) <= bound(a, b)).all()
    # sum over the batch of turned left operands, with rows one behind another and with gaps
    for layout in ("rows", "gaps"):
        ob, ov = dense(be, np.zeros((m, n), np.float32))
        at = np.ascontiguousarray(np.swapaxes(a, -1, -2))
        be.call("gemm_ranked_reduce_lhs_t", operand(be, at, layout), operand(be, b, layout), ov)
        assert (np.abs(read(ob, ov) - want.sum(0)) <= bound(a, b).sum(0)).all()
    w, bias = b[0], rng.standard_normal((1, n)).astype(np.float32)
    ob, ov = dense(be, np.zeros((batch, m, n), np.float32))
    _, wv = dense(be, w)
    be.call("gemm_ranked_matrix_rhs", operand(be, a, "rows"), wv, ov)
    be.call("add_bias_relu_rowwise_inplace", ov, dense(be, bias)[1])
    want = np.maximum(a.astype(np.float64) @ w.astype(np.float64) + bias, 0.0)
    assert (np.abs(read(ob, ov) - want) <= bound(a, w) + 2.0 ** -23 * np.abs(bias) + 2.0 ** -23 * want).all()


@pytest.mark.parametrize("m,n,k", [(300, 200, 512), (64, 96, 2048)])
def test_values_no_pair_holds(be, m, n, k):
    """Several kinds in one product, and the product after it (each kind alone: below)."""
    rng = np.random.default_rng(m)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    a[3, 7], a[5, 9], a[6, 1], a[9, :] = np.inf, np.nan, -np.inf, 0.0
    b[11, 2], a[:, 11] = 3.4028e38, np.float32(0.5)
    with np.errstate(all="ignore"):
        want = a.astype(np.float64) @ b.astype(np.float64)
    ob, ov = dense(be, np.zeros((m, n), np.float32))
    be.call("gemm", dense(be, a)[1], dense(be, b)[1], ov)
    got = read(ob, ov)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    fine = np.isfinite(want)
    assert (np.abs(got[fine] - want[fine]) <= 1e-5 * np.abs(want[fine]) + 1e-4).all()
    a[~np.isfinite(a)] = 1.0
    b[11, 2] = 1.0
    be.call("gemm", dense(be, a)[1], dense(be, b)[1], ov)  # and the next product is back on its way
    assert (np.abs(read(ob, ov) - a.astype(np.float64) @ b) <= bound(a, b)).all()


def test_small_and_tiny_values(be):
    rng = np.random.default_rng(5)
    a = (rng.standard_normal((256, 512)) * 1e-30).astype(np.float32)
    b = (rng.standard_normal((512, 256)) * 1e20).astype(np.float32)
    ob, ov = dense(be, np.zeros((256, 256), np.float32))
    be.call("gemm", dense(be, a)[1], dense(be, b)[1], ov)
    assert (np.abs(read(ob, ov) - a.astype(np.float64) @ b.astype(np.float64)) <= bound(a, b)).all()


@pytest.mark.parametrize("where", ["a", "b"])
@pytest.mark.parametrize("bits", [0x7fc00000, 0x7fffffff, 0xffffffff, 0x7f800000, 0xff800000, 0x7f7fffff, 0xff7ffff0])
@pytest.mark.parametrize("m,n,k", [(300, 200, 512), (64, 96, 2048)])
def test_one_value_no_pair_holds(be, m, n, k, bits, where):
    """One NaN (as numpy writes it, as arithmetic on the GPU does, either sign), one infinity or one value beside infinity among
    values of all lengths: where the result is NaN, where infinite, and the rest within the bound."""
    rng = np.random.default_rng(bits % 1000 + m)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    a[:, ::3], b[::2] = np.round(a[:, ::3] * 4) / 4, np.round(b[::2] * 8) / 8  # few bits, zeros among them
    one = np.uint32(bits).view(np.float32)
    if where == "a":
        a[17, 33], b[33] = one, np.where(b[33] == 0, 0.5, b[33])
        b[33, :2] = 0.5, -1.25
    else:
        b[33, 17], a[:, 33] = one, np.where(a[:, 33] == 0, 0.5, a[:, 33])
        a[:2, 33] = 0.5, -1.25
    with np.errstate(all="ignore"):
        want = a.astype(np.float64) @ b.astype(np.float64)
        within = bound(a, b)
    near = (bits & 0x7fffffff) < 0x7f800000
    if near:  # sums beside the largest number may come out either way
        sure = np.abs(want) < 3.0e38
    else:
        sure = np.ones_like(want, bool)
    ob, ov = dense(be, np.zeros((m, n), np.float32))
    be.call("gemm", dense(be, a)[1], dense(be, b)[1], ov)
    got = read(ob, ov)
    assert np.array_equal(np.isnan(got)[sure], np.isnan(want)[sure])
    fine = np.isfinite(want) & sure
    assert np.array_equal(got[sure & np.isinf(want)], want[sure & np.isinf(want)])
    # the sums in the order of k that such operands get round k times
    assert (np.abs(got[fine] - want[fine]) <= within[fine] * max(1.0, k * 2.0 ** -24 / 2.0 ** -21)).all()


@pytest.mark.parametrize("rows,k,n", [(24000, 512, 512), (40001, 130, 66)])
def test_many_rows_of_batches_with_gaps(be, rows, k, n):
    """Two left operands that do not lie one behind another, more rows each than a launch takes of a single one: the pairs of all
    of them have room. The rows' results against the same rows as one matrix, and against 64-bit sums."""
    rng = np.random.default_rng(rows)
    a = rng.standard_normal((2, rows, k)).astype(np.float32)
    w = rng.standard_normal((k, n)).astype(np.float32)
    _, av = sliced(be, a, rows + 3)
    ob, ov = dense(be, np.zeros((2, rows, n), np.float32))
    _, wv = dense(be, w)
    be.call("gemm_ranked_matrix_rhs", av, wv, ov)
    got = read(ob, ov)
    some = rng.integers(0, rows, 500)
    some[:3] = 0, rows - 1, 16384
    want = a[:, some].astype(np.float64) @ w.astype(np.float64)
    assert (np.abs(got[:, some] - want) <= bound(a[:, some], w)).all()
    ob, ov = dense(be, np.zeros((2 * rows, n), np.float32))
    be.call("gemm", dense(be, a.reshape(2 * rows, k))[1], wv, ov)
    assert (np.abs(got.reshape(2 * rows, n) - read(ob, ov)).max(0) <= 2.0 * bound(a.reshape(2 * rows, k), w).max(0)).all()


@pytest.mark.parametrize("m,n,k", [(2000, 512, 2048), (300, 200, 512)])
def test_a_product_no_pair_holds_takes_its_time_but_no_more(be, m, n, k):
    """A step that has diverged has such values everywhere: its products take up to 5 times as long as others (2000 x 512 x 2048: 42
    and 187 us), which is what fused multiply-adds take (175 us), not a multiple of that."""
    rng = np.random.default_rng(m)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    ob, ov = dense(be, np.zeros((m, n), np.float32))
    bv = dense(be, b)[1]

    def least(av):
        times = []
        for _ in range(5):
            read(ob, ov)  # (waits)
            t = time.perf_counter()
            for _ in range(30):
                be.call("gemm", av, bv, ov)
            read(ob, ov)
            times.append(time.perf_counter() - t)
        return min(times)

    usual = least(dense(be, a)[1])
    a[3, 5] = np.nan
    assert least(dense(be, a)[1]) < 9.0 * usual


def test_a_replayed_step_forgets_what_it_met(tmp_path):
    """A step of a 32-bit model, captured once and replayed: after tokens whose hidden state is not finite its products are as
    fast as before them."""
    cfg = formats.mitilix_config(512, 4000, 128, [layer(4, 32, 32, 64, 64, ff=256)], taps=2, eps=1e-5)
    w = formats.mitilix_random_weights(cfg, 3)
    # column 0 of the stream is zero but for token 7, whose feed-forward sums there leave the range
    w["embed"][:, 0] = w["pos"][:, 0] = 0.0
    w["l0.mix.o"][0] = 0.0
    w["embed"][7], w["embed"][7, 0] = 0.0, 32.0
    w["l0.mlp.up"][:16], w["l0.mlp.up"][:16, 0] = 0.0, 2.0 ** 60
    w["l0.mlp.down"][:, :16] = w["l0.mlp.down"][0] = 0.0
    w["l0.mlp.down"][0, :16] = 2.0 ** 62
    w["head"][7] = 0.0
    formats.write_model_folder(str(tmp_path / "m"), cfg, w)
    prompts = np.random.default_rng(4).integers(8, 4000, (64, 8)).astype(np.int32)
    bad = prompts.copy()
    bad[:, -1] = 7
    with ModelSession(str(tmp_path / "m"), "float32", 64) as s:
        def least_ms():
            times = []
            for _ in range(4):
                s.generate(prompts, 40)
                times.append(s.stats().device_ms)
            return min(times)

        before = least_ms()
        assert not np.isfinite(s.forward(bad)).any()
        s.generate(bad, 40)
        after = least_ms()
    assert after < 1.15 * before, (before, after)


def hits(rng, k, n):
    """A k x n matrix with a single one per column."""
    e = np.zeros((k, n), np.float32)
    e[rng.integers(0, k, n), np.arange(n)] = 1.0
    return e


@pytest.mark.parametrize("m,n,k", [(256, 200, 512), (130, 60, 1100), (700, 330, 320)])
def test_sums_of_one_term_keep_every_bit(be, m, n, k):
    """Columns of ones and zeros pick values of all lengths and sizes out of a row, unchanged; with one factor in the ones' place the
    product is a fused multiply-add's: rounded once, here within 2^-24 (half a unit in the last place) and what the sum of the parts'
    products adds, 2^-8 of that."""
    rng = np.random.default_rng(m + k)
    a = (rng.standard_normal((m, k)) * 10.0 ** rng.uniform(-30, 15, (m, k))).astype(np.float32)
    a[:, ::4] = np.ldexp(1.0 - 2.0 ** -24 * rng.integers(1, 9, a[:, ::4].shape), rng.integers(-90, 60, a[:, ::4].shape))  # below powers of two
    a[::2] *= -1.0
    e = hits(rng, k, n)
    ob, ov = dense(be, np.zeros((m, n), np.float32))
    be.call("gemm", dense(be, a)[1], dense(be, e)[1], ov)
    assert np.array_equal(read(ob, ov), a[:, e.argmax(0)])
    et, at = np.ascontiguousarray(e.T), np.ascontiguousarray(a.T)
    ob, ov = dense(be, np.zeros((n, m), np.float32))
    be.call("gemm", dense(be, et)[1], dense(be, at)[1], ov)
    assert np.array_equal(read(ob, ov), a[:, e.argmax(0)].T)
    f = e * rng.standard_normal((1, n)).astype(np.float32)
    ob, ov = dense(be, np.zeros((m, n), np.float32))
    be.call("gemm", dense(be, a)[1], dense(be, f)[1], ov)
    want = a.astype(np.float64) @ f.astype(np.float64)
    assert (np.abs(read(ob, ov) - want) <= 2.0 ** -24 * (1 + 2.0 ** -8) * np.abs(want)).all()


@pytest.mark.parametrize("m,n,k", [(200, 130, 256), (64, 300, 2048)])
@pytest.mark.parametrize("of", ["normal", "positive", "uneven"])
def test_error_not_above_sums_in_32_bits(be, m, n, k, of):
    """Against 64-bit sums, in the 2-norm: no further off than multiplied and added one after another in 32 bits."""
    rng = np.random.default_rng(k)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    if of == "positive":
        a, b = np.abs(a), np.abs(b)
    if of == "uneven":
        a, b = a * 10.0 ** rng.uniform(-5, 5, a.shape), b * 10.0 ** rng.uniform(-5, 5, b.shape)
    a, b = a.astype(np.float32), b.astype(np.float32)
    ob, ov = dense(be, np.zeros((m, n), np.float32))
    be.call("gemm", dense(be, a)[1], dense(be, b)[1], ov)
    want = a.astype(np.float64) @ b.astype(np.float64)
    plain = np.zeros((m, n), np.float32)
    for i in range(k):
        plain += a[:, i:i + 1] * b[i:i + 1]
    assert np.linalg.norm(read(ob, ov) - want) <= np.linalg.norm(plain - want)


def test_values_near_the_smallest(be):
    """Operands down to the smallest normal numbers: nothing of them is lost."""
    rng = np.random.default_rng(9)
    a = (rng.standard_normal((256, 512)) * 1e-37).astype(np.float32)
    b = (rng.standard_normal((512, 256)) * 1e17).astype(np.float32)
    ob, ov = dense(be, np.zeros((256, 256), np.float32))
    be.call("gemm", dense(be, a)[1], dense(be, b)[1], ov)
    assert (np.abs(read(ob, ov) - a.astype(np.float64) @ b.astype(np.float64)) <= bound(a, b)).all()
    a[np.abs(a) < 2.0 ** -126] = 2.0 ** -126
    e = hits(rng, 512, 256)
    be.call("gemm", dense(be, a)[1], dense(be, e)[1], ov)
    assert np.array_equal(read(ob, ov), a[:, e.argmax(0)])


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_products_of_a_first_step_share_one_allocation():
    """Each larger than the one before, as a first training step has them: the memory for their operands' parts is there from the
    first on."""
    with Backend() as fresh:
        sizes = [(256, 256, 256), (300, 512, 512), (1000, 512, 512), (2000, 512, 512), (512, 512, 2000), (2000, 2048, 512)]
        views = [(dense(fresh, np.ones((m, k), np.float32))[1], dense(fresh, np.ones((k, n), np.float32))[1],
                  dense(fresh, np.ones((m, n), np.float32))[1]) for m, n, k in sizes]
        held = set()
        for a, b, c in views:
            fresh.call("gemm", a, b, c)
            held.add(free_bytes())
    assert len(held) == 1


@pytest.mark.parametrize("order,gap,offset", [((0, 1, 2), 0, 1), ((0, 2, 1), 0, 0), ((0, 2, 1), 3, 4), ((1, 0, 2), 0, 0),
                                              ((1, 0, 2), 4, 0), ((2, 1, 0), 1, 7), ((0, 1, 2), 5, 0)])
def test_results_and_operands_in_any_order(be, order, gap, offset):
    """Batches of matrices whose three axes lie in memory in every order, with and without gaps and 16-byte rows, operands and
    results alike; what lies between the results stays as it was."""
    rng = np.random.default_rng(gap + offset)
    batch, m, n, k = 3, 130, 94, 260

    def placed(values):
        strides, at = [0, 0, 0], 1
        for axis in reversed(order):
            strides[axis] = at
            at = at * values.shape[axis] + gap
        buf = Buffer(be, (at + offset) * 4, fill=-7.0)
        view = buf.view(values.shape, [4 * x for x in strides], 4 * offset)
        buf.np_view(view)[...] = values
        buf.push()
        return buf, view

    a, b = (rng.standard_normal(x).astype(np.float32) for x in ((batch, m, k), (batch, k, n)))
    want = a.astype(np.float64) @ b.astype(np.float64)
    (_, av), (_, bv), (ob, ov) = placed(a), placed(b), placed(np.zeros((batch, m, n), np.float32))
    be.call("gemm_batched", av, bv, ov)
    assert (np.abs(read(ob, ov) - want) <= bound(a, b)).all()
    ob.np_view(ov)[...] = -7.0
    assert (ob.host.view(np.float32) == -7.0).all()
    _, wv = placed(b[:1])
    be.call("gemm_ranked_matrix_rhs", av, type(wv)(wv.ptr, wv.shape[1:], wv.strides[1:], wv.dtype, wv.device), ov)
    assert (np.abs(read(ob, ov) - a.astype(np.float64) @ b[0].astype(np.float64)) <= bound(a, b[0])).all()
    sb, sv = placed(np.zeros((1, m, n), np.float32))
    tv = type(av)(av.ptr, (batch, k, m), (av.strides[0], av.strides[2], av.strides[1]), av.dtype, av.device)
    be.call("gemm_ranked_reduce_lhs_t", tv, bv, type(sv)(sv.ptr, sv.shape[1:], sv.strides[1:], sv.dtype, sv.device))
    assert (np.abs(read(sb, sv)[0] - want.sum(0)) <= bound(a, b).sum(0)).all()
