"""The mat-mat on pairs of SMs (csrc/qmm_duo.cu) at the edges of its tiles (256 weight rows, 128 for each CTA; a multiple of 32 activation rows,
at most 256), K stages (128 values, two to a raw stage) and work shares, against the oracle with both operands rounded to f16."""
import numpy as np
import pytest
import torch

import mlx_native_b200 as mx
from oracle import oracle as orc
from tests.gpu_util import TYPES, Ctx, norm_err, normal_acts, normal_weights

pytestmark = pytest.mark.gpu
# both operands are the oracle's; the sums differ in order: sqrt(K / 16) roundings of 2^-24 of partial sums that are smaller than sum |w x|
TOL = 2e-5


@pytest.fixture(scope="module")
def ctx():
    return Ctx()


# one weight tile and a part of the next (the second CTA's half empty, or a row short); activation tiles with rows left over; K of part of a
# stage, of part of a raw stage, of an odd number of raw stages; rows at every even pitch (groups of 1, 2, 4 and 8 rows a copy)
@pytest.mark.parametrize("tname,n,k,m", [
    ("Q4_0", 8, 32, 9), ("Q4_0", 256, 96, 33), ("Q4_0", 136, 416, 31), ("Q4_0", 264, 1024, 65), ("Q4_0", 520, 2880, 257), ("Q4_0", 128, 4096, 300),
    ("Q8_0", 8, 64, 10), ("Q8_0", 120, 160, 32), ("Q8_0", 384, 1056, 97), ("Q8_0", 257, 512, 64), ("Q8_0", 504, 2048, 129),
    ("Q6_K", 8, 256, 12), ("Q6_K", 248, 768, 40), ("Q6_K", 260, 2560, 96), ("Q6_K", 513, 2048, 200), ("Q6_K", 264, 4096, 513)])
def test_dense(ctx, tname, n, k, m):
    gtype, otype = TYPES[tname]
    wq = normal_weights(n + k, n, k, otype)
    x = normal_acts(n + m, m, k)
    y = ctx.matmul(gtype, wq, x, n, k)
    assert mx.last_kernel_name() == "qmm_tc" and mx.last_mat_mat()[0] == "qmm_duo"
    y_ref, ad = orc.qmatmul(otype, wq, x, n, k, nthreads=8, f16_operands=True)
    assert norm_err(y, y_ref, ad) <= TOL
    assert np.array_equal(y.view(np.uint32), ctx.matmul(gtype, wq, x, n, k).view(np.uint32))


# more tiles than pairs of SMs: whole tiles one after another, and equal ranges that cut tiles in two
@pytest.mark.parametrize("tname,n,k,m", [("Q4_0", 20480, 256, 16), ("Q4_0", 20480, 2048, 16), ("Q6_K", 22528, 768, 40), ("Q8_0", 2048, 512, 2300)])
def test_many_tiles(ctx, tname, n, k, m):
    gtype, otype = TYPES[tname]
    part = normal_weights(k, 1024, k, otype)
    x = normal_acts(m, m, k)
    y = ctx.matmul(gtype, np.tile(part, n // 1024), x, n, k)
    assert mx.last_mat_mat()[0] == "qmm_duo"
    rows = np.r_[0:40, m - 40:m] if m > 200 else np.arange(m)
    y_ref, ad = orc.qmatmul(otype, part, x[rows], 1024, k, nthreads=8, f16_operands=True)
    for at in range(0, n, 1024):
        assert norm_err(y[rows, at:at + 1024], y_ref, ad) <= TOL
    first = y[:, :1024].view(np.uint32)   # the same weights again: where no tile is cut, the same bits
    if k == 256:
        assert all(np.array_equal(first, y[:, at:at + 1024].view(np.uint32)) for at in range(0, n, 1024))


# both kernels take the call or only the other one (weights off 16-byte boundaries): the same results within the order of the sums
@pytest.mark.parametrize("tname,n,k,m", [("Q4_0", 392, 1312, 70), ("Q8_0", 264, 1024, 130), ("Q6_K", 200, 1280, 48)])
def test_beside_the_other_kernel(ctx, tname, n, k, m):
    gtype, otype = TYPES[tname]
    wq = normal_weights(n, n, k, otype)
    big = np.zeros(wq.size + 64, np.uint8)
    big[6:6 + wq.size] = wq
    x = normal_acts(7, m, k)
    y = ctx.matmul(gtype, wq, x, n, k)
    assert mx.last_mat_mat()[0] == "qmm_duo"
    z = ctx.matmul(gtype, wq, x, n, k, weight_buf=ctx.buf(big, mx.DType.U8).slice_view(6, wq.size))
    assert mx.last_mat_mat()[0] == "qmm_tc"
    y_ref, ad = orc.qmatmul(otype, wq, x, n, k, nthreads=8, f16_operands=True)
    assert norm_err(y, y_ref, ad) <= TOL and norm_err(z, y_ref, ad) <= TOL


def sum_error(y, otype, wq, x, n, k):
    """Relative error of the sums: against 64 bits of the operands that both kernels multiply, rounded to f16."""
    f16 = lambda a: torch.tensor(np.ascontiguousarray(a, np.float32)).cuda().half().double()
    ref = f16(x) @ f16(orc.dequantize(otype, wq).reshape(n, k)).T
    return float((torch.tensor(y).cuda().double() - ref).norm() / ref.norm())


# An accumulator's chain of additions is off by 1.2e-9 of the result for each K value, and no chain may be longer than those of the kernel on
# single SMs (which takes weights off 16-byte boundaries); chains of 512 values, 6.1e-7, count as short.  One, two and four accumulators; whole
# tiles, halves and ranges.
CHAINS = [("Q4_0", 4096, 4096, 512), ("Q4_0", 4096, 4096, 333), ("Q8_0", 1024, 4096, 60), ("Q6_K", 1024, 4096, 96), ("Q4_0", 2688, 1792, 585),
          ("Q8_0", 6464, 7680, 782), ("Q4_0", 12288, 2048, 512), ("Q6_K", 256, 768, 1000)]
SHORT = 6.2e-7


def other_kernel(ctx, gtype, wq, x, n, k):
    big = np.zeros(wq.size + 64, np.uint8)
    big[6:6 + wq.size] = wq.reshape(-1)
    y = ctx.matmul(gtype, wq, x, n, k, weight_buf=ctx.buf(big, mx.DType.U8).slice_view(6, wq.size))
    assert mx.last_mat_mat()[0] == "qmm_tc"
    return y


@pytest.mark.parametrize("tname,n,k,m", CHAINS)
def test_sums_are_as_exact_as_on_single_sms(ctx, tname, n, k, m):
    gtype, otype = TYPES[tname]
    wq, x = normal_weights(n + k, n, k, otype), normal_acts(m, m, k)
    other = sum_error(other_kernel(ctx, gtype, wq, x, n, k), otype, wq, x, n, k)
    y = ctx.matmul(gtype, wq, x, n, k)
    assert mx.last_mat_mat()[0] == "qmm_duo"
    assert sum_error(y, otype, wq, x, n, k) <= max(1.05 * other, SHORT)
    assert np.array_equal(y.view(np.uint32), ctx.matmul(gtype, wq, x, n, k).view(np.uint32))


# products that travel together, tiles of at most 192 rows: chains of half of K
@pytest.mark.parametrize("ns,k,m", [((4096, 1024, 1024), 4096, 512), ((5120, 640, 640), 2560, 300), ((9216, 9216), 2048, 100)])
def test_sums_of_one_group(ctx, ns, k, m):
    gtype, otype = TYPES["Q4_0"]
    d, x = ctx.device, normal_acts(m, m, k)
    ws = [normal_weights(i, n, k, otype) for i, n in enumerate(ns)]
    xb, bufs = ctx.buf(x, mx.DType.F32), [(ctx.buf(w, mx.DType.U8), d.alloc_buffer(m * n * 4, mx.DType.F32)) for w, n in zip(ws, ns)]
    enc = d.command_encoder()
    mx.reset_counters()
    for (wb, yb), n in zip(bufs, ns):
        mx.quantized_matmul_ggml(enc, ctx.registry, d, xb, wb, yb, mx.GgmlQuantizedMatmulParams(m, n, k, gtype))
    enc.commit_and_wait()
    assert mx.kernel_launch_count() == 2
    for (_, yb), w, n in zip(bufs, ws, ns):
        assert sum_error(yb.as_slice(np.float32).reshape(m, n), otype, w, x, n, k) <= 1.3e-9 * k / 2


def test_infinities_stay_in_their_row(ctx):
    gtype, otype = TYPES["Q8_0"]
    n, k, m = 264, 512, 48
    wq = normal_weights(3, n, k, otype)
    x = normal_acts(3, m, k)
    x[5, 17], x[40, 300] = np.inf, np.nan
    y = ctx.matmul(gtype, wq, x, n, k)
    bad = np.zeros(m, bool)
    bad[[5, 40]] = True
    assert np.isfinite(y[~bad]).all() and not np.isfinite(y[bad]).any()   # (no weight of these is zero)
    y_ref, ad = orc.qmatmul(otype, wq, x[~bad], n, k, nthreads=4, f16_operands=True)
    assert norm_err(y[~bad], y_ref, ad) <= TOL


def test_products_of_one_group_share_a_launch(ctx):
    """Between two barriers: three products of the same activations are packed once and leave as one kernel; one of another type and one of
    other activations do not join them; a dependent one starts a new group.  Row counts that leave part of a tile between two products."""
    d, m, k = ctx.device, 70, 1024
    gtype, otype = TYPES["Q4_0"]
    x, x2 = normal_acts(1, m, k), normal_acts(2, m, k)
    ns = (264, 512, 136)
    ws = [normal_weights(i, n, k, otype) for i, n in enumerate(ns)]
    w8 = normal_weights(9, 256, k, orc.Q8_0)
    wd = normal_weights(8, 40, 512, otype)
    xb, x2b = ctx.buf(x, mx.DType.F32), ctx.buf(x2, mx.DType.F32)
    P = mx.GgmlQuantizedMatmulParams
    out = lambda n: d.alloc_buffer(m * n * 4, mx.DType.F32)
    ys, y8, yx, yd = [out(n) for n in ns], out(256), out(264), out(40)
    for capture in (False, True):
        enc = d.command_encoder()

        def encode():
            for w, y, n in zip(wbufs, ys, ns):
                mx.quantized_matmul_ggml(enc, ctx.registry, d, xb, w, y, P(m, n, k, gtype))
            mx.quantized_matmul_ggml(enc, ctx.registry, d, xb, w8b, y8, P(m, 256, k, TYPES["Q8_0"][0]))
            mx.quantized_matmul_ggml(enc, ctx.registry, d, x2b, wbufs[0], yx, P(m, 264, k, gtype))
            mx.quantized_matmul_ggml(enc, ctx.registry, d, ys[1], wdb, yd, P(m, 40, 512, gtype))

        wbufs, w8b, wdb = [ctx.buf(w, mx.DType.U8) for w in ws], ctx.buf(w8, mx.DType.U8), ctx.buf(wd, mx.DType.U8)
        mx.reset_counters()
        encode()
        enc.commit_and_wait()
        assert mx.kernel_launch_count() == 2 * 4
        if capture:
            enc.begin_capture()
            encode()
            graph = enc.end_capture()
            graph.launch(enc)
            enc.commit_and_wait()
        refs = [(y, n, w, otype, x, k) for y, n, w in zip(ys, ns, ws)] + [(y8, 256, w8, orc.Q8_0, x, k), (yx, 264, ws[0], otype, x2, k)]
        for y, n, w, o, xx, kk in refs:
            y_ref, ad = orc.qmatmul(o, w, xx, n, kk, nthreads=4, f16_operands=True)
            assert norm_err(y.as_slice(np.float32).reshape(m, n), y_ref, ad) <= TOL
        mid = ys[1].as_slice(np.float32).reshape(m, 512).copy()
        y_ref, ad = orc.qmatmul(otype, wd, mid, 40, 512, nthreads=4, f16_operands=True)
        assert norm_err(yd.as_slice(np.float32).reshape(m, 40), y_ref, ad) <= TOL


def test_products_of_one_group_over_shared_ranges(ctx):
    """Two products whose tiles together are more than the pairs of SMs, cut into equal ranges: the zeroed tiles are those of both."""
    gtype, otype = TYPES["Q4_0"]
    d, m, n, k = ctx.device, 16, 10240, 2048
    part = normal_weights(4, 1024, k, otype)
    x = normal_acts(4, m, k)
    y_ref, ad = orc.qmatmul(otype, part, x, 1024, k, nthreads=8, f16_operands=True)
    xb, wb = ctx.buf(x, mx.DType.F32), ctx.buf(np.tile(part, n // 1024), mx.DType.U8)
    ys = [ctx.buf(np.full(m * n, 7, np.float32), mx.DType.F32) for _ in range(2)]
    enc = d.command_encoder()
    mx.reset_counters()
    for y in ys:
        mx.quantized_matmul_ggml(enc, ctx.registry, d, xb, wb, y, mx.GgmlQuantizedMatmulParams(m, n, k, gtype))
    enc.commit_and_wait()
    assert mx.kernel_launch_count() == 2
    for y in ys:
        got = y.as_slice(np.float32).reshape(m, n)
        for at in range(0, n, 1024):
            assert norm_err(got[:, at:at + 1024], y_ref, ad) <= TOL


ROUTED = [
    # (type, n, k): 264 and 520 weight rows leave a pair of SMs half or almost empty; K tails of 32; Q4_0 with 261 rows has no groups of
    # rows that start on 16 bytes, so the other kernel takes it
    ("Q4_0", 264, 288), ("Q4_0", 261, 288), ("Q4_0", 520, 2048), ("Q8_0", 264, 544), ("Q8_0", 96, 32),
    ("Q6_K", 520, 768), ("Q6_K", 256, 256), ("Q4_K", 264, 768), ("Q4_K", 1032, 256),
]


@pytest.mark.parametrize("tname,n,k", ROUTED)
def test_routed_tiles(ctx, tname, n, k):
    """Experts with no rows, one, either side of a CTA's half of a tile, of a whole tile and of two, and a row whose id names no expert."""
    gtype, otype = (mx.GgmlType.Q4_K, orc.Q4_K) if tname == "Q4_K" else TYPES[tname]
    counts = [0, 1, 32, 33, 63, 64, 65, 0, 130]
    E, m = len(counts), sum(counts) + 1
    ids = np.random.default_rng(n + k).permutation(np.concatenate([np.repeat(np.arange(E), counts), [E + 7]])).astype(np.uint32)
    ws = [normal_weights(50 + e, n, k, otype) for e in range(E)]
    stride = (ws[0].size + 15) // 16 * 16 + 48
    stack = np.zeros(E * stride, np.uint8)
    for e, w in enumerate(ws):
        stack[e * stride:e * stride + w.size] = w.reshape(-1)
    x = normal_acts(3, m, k)
    d = ctx.device
    xb, wb, ib = ctx.buf(x, mx.DType.F32), ctx.buf(stack, mx.DType.U8), ctx.buf(ids, mx.DType.U32)
    yb = ctx.buf(np.full(m * n, 7, np.float32), mx.DType.F32)
    enc = d.command_encoder()
    mx.quantized_matmul_id_ggml(enc, ctx.registry, d, xb, wb, ib, yb, mx.GgmlQuantizedMatmulIdParams(m, 1, n, k, E, stride, gtype))
    enc.commit_and_wait()
    y = yb.as_slice(np.float32).reshape(m, n)
    for e in range(E):
        rows = np.nonzero(ids == e)[0]
        if rows.size:
            y_ref, ad = orc.qmatmul(otype, ws[e], x[rows], n, k, nthreads=4, f16_operands=True)
            assert norm_err(y[rows], y_ref, ad) <= TOL
    assert not y[ids == E + 7].any()
    assert mx.last_mat_mat() == ("qmm_tc_id" if n == 261 else "qmm_duo_id", 64)


def test_routed_layer_with_one_result_buffer(ctx):
    """gate and up written to the same buffer: up's product is what stays, so it may not run beside the other one."""
    d, T, E, top_k, hidden, ffn = ctx.device, 256, 8, 2, 512, 512
    gtype, otype = TYPES["Q4_0"]
    gate, up, down = (np.concatenate([normal_weights(at + e, 512, 512, otype) for e in range(E)]) for at in (0, 20, 40))
    ids = np.random.default_rng(1).permuted(np.tile(np.arange(E), (T, 1)), axis=1)[:, :top_k].astype(np.uint32).reshape(-1)
    xb, ib = ctx.buf(normal_acts(5, T, hidden), mx.DType.F32), ctx.buf(ids, mx.DType.U32)
    p = mx.MoeFfnLayerParams(T, top_k, hidden, ffn, E, gtype, gtype, gtype, *([gate.size // E] * 3))
    got = []
    for one in (True, False):
        wg, wu, wd = (ctx.buf(w, mx.DType.U8) for w in (gate if one else up, up, down))
        yu, yd = (d.alloc_buffer(T * top_k * ffn * 4, mx.DType.F32) for _ in range(2))
        yg = yu if one else d.alloc_buffer(T * top_k * ffn * 4, mx.DType.F32)
        enc = d.command_encoder()
        mx.moe_ffn_layer(enc, ctx.registry, d, xb, ib, wg, wu, wd, yg, yu, yd, p)
        enc.commit_and_wait()
        got.append((yu.as_slice(np.float32).copy(), yd.as_slice(np.float32).copy()))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("gate_off", [0, 6])
def test_routed_layer_with_the_result_over_weights(ctx, gate_off):
    """up's result over gate's weights, which the gate product has to have read by then.  With gate's weights off 16-byte boundaries the kernel
    ahead of up's is the one on single SMs."""
    d, T, E, top_k, hidden, ffn = ctx.device, 256, 8, 2, 512, 512
    gtype, otype = TYPES["Q4_0"]
    gate, up, down = (np.concatenate([normal_weights(at + e, 512, 512, otype) for e in range(E)]).reshape(-1) for at in (0, 20, 40))
    ids = np.random.default_rng(1).permuted(np.tile(np.arange(E), (T, 1)), axis=1)[:, :top_k].astype(np.uint32).reshape(-1)
    xb, ib = ctx.buf(normal_acts(5, T, hidden), mx.DType.F32), ctx.buf(ids, mx.DType.U32)
    p = mx.MoeFfnLayerParams(T, top_k, hidden, ffn, E, gtype, gtype, gtype, *([gate.size // E] * 3))
    result, got = T * top_k * ffn * 4, []
    for over in (True, False):
        big = np.zeros(max(gate.size + 64, result), np.uint8)
        big[gate_off:gate_off + gate.size] = gate
        both = ctx.buf(big, mx.DType.U8)
        wg, wu, wd = both.slice_view(gate_off, gate.size), ctx.buf(up, mx.DType.U8), ctx.buf(down, mx.DType.U8)
        yu = both.slice_view(0, result) if over else d.alloc_buffer(result, mx.DType.F32)
        yg, yd = d.alloc_buffer(result, mx.DType.F32), d.alloc_buffer(T * top_k * hidden * 4, mx.DType.F32)
        enc = d.command_encoder()
        mx.moe_ffn_layer(enc, ctx.registry, d, xb, ib, wg, wu, wd, yg, yu, yd, p)
        enc.commit_and_wait()
        assert mx.last_mat_mat()[0] == "qmm_duo_id"
        got.append([b.as_slice(np.float32).copy() for b in (yg, yu, yd)])
    assert all(np.array_equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("capture", [False, True])
def test_waiting_products_beside_the_other_lane(ctx, capture):
    """A group of two products that wait, then work that starts at once on the other lane; the next groups write over what these read."""
    gtype, otype = TYPES["Q4_0"]
    d, m, n = ctx.device, 40, 512
    ws = [normal_weights(i, n, n, otype) for i in range(2)]
    wbufs = [ctx.buf(w, mx.DType.U8) for w in ws]
    a, gate, up = normal_acts(1, m, n), normal_acts(2, m, n), normal_acts(3, m, n)
    bufs = {k: ctx.buf(v, mx.DType.F32) for k, v in (("a", a), ("g", gate), ("u", up))}
    for k in ("b", "c", "s", "t"):
        bufs[k] = ctx.buf(np.zeros((m, n), np.float32), mx.DType.F32)
    p = mx.GgmlQuantizedMatmulParams(m, n, n, gtype)
    enc = d.command_encoder()

    def encode():
        for _ in range(4):
            for w, y in zip(wbufs, "bc"):
                mx.quantized_matmul_ggml(enc, ctx.registry, d, bufs["a"], w, bufs[y], p)          # wait for one another
            mx.silu_mul(enc, ctx.registry, d, bufs["g"], bufs["u"], bufs["s"], m * n)              # other lane
            mx.silu_mul(enc, ctx.registry, d, bufs["s"], bufs["u"], bufs["t"], m * n)              # conflict: a new group
            mx.quantized_matmul_ggml(enc, ctx.registry, d, bufs["t"], wbufs[0], bufs["s"], p)      # reads t, writes over s
            mx.quantized_matmul_ggml(enc, ctx.registry, d, bufs["c"], wbufs[1], bufs["b"], p)      # reads c, writes over b

    encode()
    enc.commit_and_wait()
    if capture:
        for k in ("b", "c", "s", "t"):
            bufs[k].as_mut_slice(np.float32)[:] = 0
            mx.silu_mul(enc, ctx.registry, d, bufs[k], bufs[k], bufs["t"], m * n)   # (uploaded before the recording)
        enc.commit_and_wait()
        enc.begin_capture()
        encode()
        graph = enc.end_capture()
        graph.launch(enc)
        enc.commit_and_wait()
    get = lambda k: bufs[k].as_slice(np.float32).reshape(m, n).copy()
    silu = lambda g, u: (g / (1 + np.exp(-g.astype(np.float64))) * u).astype(np.float32)
    t, c = get("t"), get("c")
    assert np.allclose(t, silu(silu(gate, up), up), rtol=1e-5, atol=1e-6)
    for got, x, w in ((c, a, ws[1]), (get("b"), c, ws[1]), (get("s"), t, ws[0])):
        y_ref, ad = orc.qmatmul(otype, w, x, n, n, nthreads=4, f16_operands=True)
        assert norm_err(got, y_ref, ad) <= TOL


# The kernel on single SMs keeps its tiles of 16 rows (a long K, so that converting for each tile is what a call takes), which that on
# pairs of SMs does not have.
@pytest.mark.parametrize("tname,n,k,m", [("Q4_0", 256, 10496, 45), ("Q8_0", 320, 10496, 93)])
def test_tiles_of_16_rows_on_single_sms(ctx, tname, n, k, m):
    gtype, otype = TYPES[tname]
    wq, x = normal_weights(n, n, k, otype), normal_acts(m, m, k)
    y = other_kernel(ctx, gtype, wq, x, n, k)
    assert mx.last_mat_mat() == ("qmm_tc", 16)
    y_ref, ad = orc.qmatmul(otype, wq, x, n, k, nthreads=8, f16_operands=True)
    assert norm_err(y, y_ref, ad) <= TOL
    ctx.matmul(gtype, wq, x, n, k)
    assert mx.last_mat_mat()[0] == "qmm_duo"
