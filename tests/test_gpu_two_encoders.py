"""Command buffers of several encoders run in the order in which they were encoded, also where an encoder has put off the launch of its products
until it knows what they can share a launch with."""
import threading

import numpy as np
import pytest

import mlx_native_b200 as mx
from oracle import oracle as orc
from tests.gpu_util import MM_TOL, Ctx, norm_err, normal_acts, normal_weights

pytestmark = pytest.mark.gpu
G = mx.GgmlType
# products whose launch is put off: register-level mat-vec, mat-mat on pairs of SMs, Q4_K of many rows, split mat-vec (weights off 16 bytes)
KINDS = {"mat-vec": (G.Q8_0, orc.Q8_0, 1, 0), "mat-mat": (G.Q4_0, orc.Q4_0, 16, 0), "wide": (G.Q4_K, orc.Q4_K, 12, 0), "split": (G.Q4_0, orc.Q4_0, 2, 6)}
N, K = 1024, 1024


@pytest.fixture(scope="module")
def ctx():
    return Ctx()


class Product:
    """y = x W, with x and y of the same size, so that results can be operands."""

    def __init__(self, ctx, kind, seed=0):
        self.ctx, (self.gtype, self.otype, self.m, off) = ctx, KINDS[kind]
        wq = normal_weights(seed + 5, N, K, self.otype).reshape(-1)
        big = np.zeros(wq.size + 64, np.uint8)
        big[off:off + wq.size] = wq
        self.wq, self.x = wq, normal_acts(seed + 1, self.m, K)
        self.w = ctx.buf(big, mx.DType.U8).slice_view(off, wq.size)
        self.xb, self.yb = ctx.buf(self.x, mx.DType.F32), ctx.buf(np.zeros((self.m, N), np.float32), mx.DType.F32)

    def encode(self, enc, x=None, y=None):
        c = self.ctx
        mx.quantized_matmul_ggml(enc, c.registry, c.device, x or self.xb, self.w, y or self.yb, mx.GgmlQuantizedMatmulParams(self.m, N, K, self.gtype))

    def check(self, y, x=None):
        y_ref, ad = orc.qmatmul(self.otype, self.wq, self.x if x is None else x, N, K, nthreads=4)
        assert norm_err(np.asarray(y).reshape(self.m, N), y_ref, ad) <= MM_TOL


def silu(g, u):
    g = g.astype(np.float64)
    return (g / (1 + np.exp(-g)) * u).astype(np.float32)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("first", ["writer", "reader"])
def test_result_read_through_another_encoder(ctx, kind, first):
    """A: y = x W; B: out = silu(y) u.  Whichever is committed first."""
    p = Product(ctx, kind)
    d, u = ctx.device, normal_acts(9, p.m, N)
    ub, out = ctx.buf(u, mx.DType.F32), ctx.buf(np.zeros((p.m, N), np.float32), mx.DType.F32)
    a, b = d.command_encoder(), d.command_encoder()
    p.encode(a)
    mx.silu_mul(b, ctx.registry, d, p.yb, ub, out, p.m * N)
    for enc in ((a, b) if first == "writer" else (b, a)):
        enc.commit_and_wait()
    y = p.yb.as_slice(np.float32).copy()
    p.check(y)
    ref = silu(y.reshape(p.m, N), u)
    assert np.allclose(out.as_slice(np.float32).reshape(p.m, N), ref, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("kind", KINDS)
def test_operand_written_through_another_encoder(ctx, kind):
    """A: y = x W; B: x = silu(g) u.  y is the product of the x before."""
    p = Product(ctx, kind)
    d, g, u = ctx.device, normal_acts(8, p.m, K), normal_acts(9, p.m, K)
    gb, ub = ctx.buf(g, mx.DType.F32), ctx.buf(u, mx.DType.F32)
    a, b = d.command_encoder(), d.command_encoder()
    p.encode(a)
    mx.silu_mul(b, ctx.registry, d, gb, ub, p.xb, p.m * K)
    b.commit_and_wait()
    a.commit_and_wait()
    p.check(p.yb.as_slice(np.float32))
    assert np.allclose(p.xb.as_slice(np.float32).reshape(p.m, K), silu(g, u), rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("how", ["host", "encoder", "encoder after commit"])
def test_operand_that_several_encoders_still_have_to_read(ctx, kind, how):
    """A and B: products of the same x, both put off, and C reads it too; then x changes."""
    p = Product(ctx, kind)
    d, g, u = ctx.device, normal_acts(8, p.m, K), normal_acts(9, p.m, K)
    gb, ub, tb = ctx.buf(g, mx.DType.F32), ctx.buf(u, mx.DType.F32), d.alloc_buffer(p.m * K * 4, mx.DType.F32)
    y2 = ctx.buf(np.zeros((p.m, N), np.float32), mx.DType.F32)
    a, b, c, e = (d.command_encoder() for _ in range(4))
    p.encode(a)
    p.encode(b, y=y2)
    mx.silu_mul(c, ctx.registry, d, p.xb, ub, tb, p.m * K)
    if how == "encoder after commit":
        for enc in (a, b, c):
            enc.commit()
    if how == "host":
        p.xb.as_mut_slice(np.float32)[:] = 0
    else:
        mx.silu_mul(e, ctx.registry, d, gb, ub, p.xb, p.m * K)
        e.commit()
    for enc in (c, b, a, e):
        enc.commit_and_wait()
    for y in (p.yb, y2):
        p.check(y.as_slice(np.float32))
    assert np.allclose(tb.as_slice(np.float32).reshape(p.m, K), silu(p.x, u), rtol=1e-5, atol=1e-6)


def test_chain_over_two_encoders_in_turn(ctx):
    """Each product reads what the other encoder's product before it writes."""
    p = Product(ctx, "mat-mat")
    d = ctx.device
    bufs = [p.xb] + [ctx.buf(np.zeros((p.m, K), np.float32), mx.DType.F32) for _ in range(6)]
    encs = [d.command_encoder(), d.command_encoder()]
    for i in range(6):
        p.encode(encs[i & 1], x=bufs[i], y=bufs[i + 1])
    for enc in reversed(encs):
        enc.commit_and_wait()
    got = [b.as_slice(np.float32).reshape(p.m, K).copy() for b in bufs]
    for i in range(6):
        p.check(got[i + 1], x=got[i])


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("how", ["host", "encoder", "commit", "dropped"])
def test_product_encoded_between_commit_and_wait(ctx, kind, how):
    """The wait is for what was committed: a product that has been encoded since keeps its buffers and its place."""
    p, q = Product(ctx, kind), Product(ctx, kind, seed=60)
    d = ctx.device
    enc, other = d.command_encoder(), d.command_encoder()
    p.encode(enc)
    enc.commit()
    q.encode(enc)
    if how == "dropped":   # nobody but the encoder holds the operand's and the weights' buffers any more
        q.xb = q.w = None
    enc.wait_until_completed()
    p.check(p.yb.as_slice(np.float32))
    if how == "host":
        q.xb.as_mut_slice(np.float32)[:] = 0
    elif how == "encoder":
        mx.silu_mul(other, ctx.registry, d, p.yb, p.yb, q.xb, q.m * K)
        other.commit_and_wait()
    elif how == "dropped":
        fill = [d.alloc_buffer(q.m * K * 4, mx.DType.F32) for _ in range(4)] + [d.alloc_buffer(q.wq.size + 64, mx.DType.U8) for _ in range(4)]
        for b in fill:
            b.as_mut_slice(np.uint8)[:] = 255
    enc.commit_and_wait()
    q.check(q.yb.as_slice(np.float32))


def test_threads_with_an_encoder_each(ctx):
    """Two threads share weights; a third one looks at results and at an operand while the others encode."""
    d = ctx.device
    shared = Product(ctx, "mat-mat")
    jobs, failed, stop = [Product(ctx, "mat-mat", seed) for seed in (20, 40)], [], threading.Event()
    for j in jobs:
        j.w, j.wq = shared.w, shared.wq

    def work(j):
        try:
            reg, enc = mx.KernelRegistry.new(), d.command_encoder()
            for _ in range(60):
                for _ in range(3):
                    mx.quantized_matmul_ggml(enc, reg, d, j.xb, j.w, j.yb, mx.GgmlQuantizedMatmulParams(j.m, N, K, j.gtype))
                enc.commit_and_wait()
        except Exception as ex:   # (shown by the test's own thread)
            failed.append(ex)

    def look():
        try:
            while not stop.is_set():
                for j in jobs:
                    j.yb.as_slice(np.float32)
                shared.w.as_slice(np.uint8)
        except Exception as ex:
            failed.append(ex)

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    watcher = threading.Thread(target=look)
    for t in threads + [watcher]:
        t.start()
    for t in threads:
        t.join(120)
    stop.set()
    watcher.join(120)
    assert not failed and not any(t.is_alive() for t in threads + [watcher])
    for j in jobs:
        j.check(j.yb.as_slice(np.float32))
