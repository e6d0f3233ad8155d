"""One and two activation rows on the split mat-vec (csrc/qmv_split.cuh: codes and activation digits as 8-bit integers), and how its tiles are shared
out, against the oracle."""
import numpy as np
import pytest

import mlx_native_b200 as mx
from oracle import oracle as orc
from tests.gpu_util import MV_TOL, TYPES, Ctx, norm_err, normal_acts, normal_weights

pytestmark = pytest.mark.gpu
ALL = dict(TYPES, Q4_K=(mx.GgmlType.Q4_K, orc.Q4_K))


@pytest.fixture(scope="module")
def ctx():
    mx.set_option("qmv", "split")
    yield Ctx()
    mx.set_option("qmv", "auto")


# every other row on a 16-byte boundary (tensor copies of the even and the odd rows) with an even and an odd number of rows, which leaves row
# copies; chunks of one to four tiles, a share that crosses from one chunk to the next, ranks without units, K of one unit and of half a unit
@pytest.mark.parametrize("tname,n,k", [("Q4_0", 50, 2176), ("Q4_0", 51, 2176), ("Q8_0", 34, 640), ("Q8_0", 33, 640), ("Q6_K", 70, 5120),
                                       ("Q6_K", 4802, 1024), ("Q4_0", 6144, 256), ("Q4_0", 10000, 512), ("Q8_0", 9520, 256), ("Q6_K", 24000, 512),
                                       ("Q4_K", 15000, 256), ("Q4_0", 33, 64), ("Q8_0", 17, 32), ("Q4_K", 96, 9216)])
@pytest.mark.parametrize("m", [1, 2])
def test_shapes(ctx, tname, n, k, m):
    gtype, otype = ALL[tname]
    wq = normal_weights(n + k, n, k, otype)
    x = normal_acts(n + m, m, k)
    y = ctx.matmul(gtype, wq, x, n, k)
    assert mx.last_kernel_name() == "qmv_split"
    y_ref, ad = orc.qmatmul(otype, wq, x, n, k, nthreads=8)
    assert norm_err(y, y_ref, ad) <= MV_TOL
    assert np.array_equal(y.view(np.uint32), ctx.matmul(gtype, wq, x, n, k).view(np.uint32))


# More than 64 units (64 values of K) on a rank, 32 with two rows: activations beyond the passes that stay in registers are loaded again, in digits and
# (with a large activation) in halves.  80 to 84 units on each of eight ranks; rows on 16-byte boundaries, every other one, and by row copies.
@pytest.mark.parametrize("tname,n,k", [("Q4_0", 34, 40960), ("Q4_0", 34, 41088), ("Q4_0", 33, 41088), ("Q8_0", 34, 40960), ("Q8_0", 18, 41088),
                                       ("Q8_0", 17, 41088), ("Q6_K", 34, 40960), ("Q6_K", 34, 41984), ("Q6_K", 33, 41984), ("Q4_K", 34, 40960)])
@pytest.mark.parametrize("m", [1, 2])
@pytest.mark.parametrize("large", [0, 1e4])
def test_long_rows(ctx, tname, n, k, m, large):
    gtype, otype = ALL[tname]
    wq = normal_weights(n + k, n, k, otype)
    x = normal_acts(n + m, m, k)
    if large:
        x[-1, ::513] = large
    y = ctx.matmul(gtype, wq, x, n, k)
    assert mx.last_kernel_name() == "qmv_split"
    y_ref, ad = orc.qmatmul(otype, wq, x, n, k, nthreads=8)
    assert norm_err(y, y_ref, ad) <= MV_TOL


@pytest.mark.parametrize("tname", sorted(ALL))
@pytest.mark.parametrize("m", [1, 2])
@pytest.mark.parametrize("shapes", [[(5000, 2048), (70, 256), (3000, 2048), (2600, 1024)], [(100, 4096), (33, 512), (16, 4096), (257, 1024)]])
@pytest.mark.parametrize("large", [(), (1,), (0, 2)])
def test_products_of_different_activations_in_one_launch(ctx, tname, m, shapes, large):
    """Shares that cross from one product to the next take that one's activations, in digits or halves; of the products of few rows, some ranks of
    a cluster have no units of the shorter ones."""
    gtype, otype = ALL[tname]
    d = ctx.device
    if tname == "Q6_K":
        shapes = [(n, max(k, 2048)) for n, k in shapes]   # (rows on 16-byte boundaries: one launch)
    ws = [normal_weights(i, n, k, otype) for i, (n, k) in enumerate(shapes)]
    xs = [normal_acts(i, m, k) * np.float32(4.0 ** i) for i, (n, k) in enumerate(shapes)]
    for i in large:
        xs[i][:, ::300] *= np.float32(1e4)
    bufs = [(ctx.buf(x, mx.DType.F32), ctx.buf(w, mx.DType.U8), d.alloc_buffer(m * n * 4, mx.DType.F32)) for x, w, (n, k) in zip(xs, ws, shapes)]
    mx.reset_counters()
    enc = d.command_encoder()
    for (xb, wb, yb), (n, k) in zip(bufs, shapes):
        mx.quantized_matmul_ggml(enc, ctx.registry, d, xb, wb, yb, mx.GgmlQuantizedMatmulParams(m, n, k, gtype))
    enc.commit_and_wait()
    assert mx.last_kernel_name() == "qmv_split" and mx.kernel_launch_count() == 1
    for (xb, wb, yb), w, x, (n, k) in zip(bufs, ws, xs, shapes):
        y_ref, ad = orc.qmatmul(otype, w, x, n, k, nthreads=8)
        assert norm_err(yb.as_slice(np.float32).reshape(m, n), y_ref, ad) <= MV_TOL


# Products of codes and digits and the sums of a block are exact; digits leave out less than 2^-29 of the largest activation of a warp's share, which
# for normal activations is 2^-27 of one, and the f32 sums of a result have at most a few dozen terms one after another: 1.5e-7 (2^-23 = 1.2e-7).
@pytest.mark.parametrize("tname", sorted(ALL))
@pytest.mark.parametrize("outliers", [False, True])
def test_error_against_64_bits(ctx, tname, outliers):
    gtype, otype = ALL[tname]
    n, k = 700, 4096
    wq = normal_weights(n, n, k, otype)
    w = orc.dequantize(otype, wq).reshape(n, k).astype(np.float64)
    for m in (1, 2):
        x = normal_acts(m, m, k)
        if outliers:
            x[:, ::97] *= 300
        y, ref = ctx.matmul(gtype, wq, x, n, k), x.astype(np.float64) @ w.T
        assert np.linalg.norm(y - ref) <= 1.5e-7 * np.linalg.norm(ref)


def same_scale(tname, k):
    """Which values share a power of two where a share of K is taken in f16 halves: the 32 of a block (Q6_K: of two 16-value groups, 32 apart)."""
    i = np.arange(k)
    return i // 128 * 4 + i // 16 % 2 * 2 + i % 128 // 64 if tname == "Q6_K" else i // 32


# Activations far larger than the others whose weights are zero: what is left of a result are the small ones.  For each output, of sum |w| |x|:
# 2e-7 for the sums (some 30 additions one after another, each 2^-24 of a partial sum, which random signs keep below a tenth of that sum), and the
# values beside a large one R lose 2^-38 R at most, halves under one power of two having a last place of 2^-24 of which the largest takes 2^13 or more.
# (Q4_K: a zero weight is code times scale less offset, in f32: another 2^-21 R of the largest weight of its sub-block.)
@pytest.mark.parametrize("tname", sorted(ALL))
@pytest.mark.parametrize("large", ["some", "stretches"])
@pytest.mark.parametrize("R", [30, 100, 1e3, 1e4, 1e5, 1e6, 1e8])
def test_small_activations_beside_large_ones(ctx, tname, large, R):
    gtype, otype = ALL[tname]
    n, k = 600, 4096
    rng = np.random.default_rng(int(R))
    at = np.arange(8) * 512 + rng.integers(0, 512, 8) if large == "some" else np.flatnonzero(np.arange(k) // 256 % 2)
    wf = (rng.standard_normal((n, k)) * 0.02).astype(np.float32)
    if tname == "Q4_K":
        wf = np.abs(wf)          # (a sub-block of positive weights has no offset, so that zero is among its values)
    wf[:, at] = 0
    wq = orc.quantize(otype, wf)
    w = orc.dequantize(otype, wq).reshape(n, k).astype(np.float64)
    assert not w[:, at].any()
    x = normal_acts(1, 2, k)
    x[0, at] = x[0, at] * np.float32(R) if large == "stretches" else np.float32(R) * np.sign(x[0, at])
    top = np.abs(x[0, at]).max()
    group = same_scale(tname, k)
    beside = np.abs(w[:, np.isin(group, group[at])]).sum(1)
    for rows in (x[:1], x):
        y = ctx.matmul(gtype, wq, rows, n, k)
        assert mx.last_kernel_name() == "qmv_split"
        for r, row in enumerate(rows):
            bound = 2e-7 * (np.abs(w) @ np.abs(row).astype(np.float64))
            if r == 0:
                bound += 2.0 ** -38 * top * beside
                if tname == "Q4_K":
                    bound += 2.0 ** -21 * top * np.abs(w).reshape(n, k // 32, 32).max(2)[:, at // 32].sum(1)
            assert np.all(np.abs(y[r] - w @ row.astype(np.float64)) <= bound)


def test_zero_and_tiny_rows(ctx):
    """A row of zeros, of the smallest numbers there are, and one of them among zeros: the scale takes two powers of two."""
    gtype, otype = TYPES["Q8_0"]
    n, k = 40, 1024
    wq = normal_weights(3, n, k, otype)
    w = orc.dequantize(otype, wq).reshape(n, k).astype(np.float64)
    x = np.zeros((3, k), np.float32)
    x[1] = normal_acts(1, 1, k) * np.float32(1e-37)
    x[2, 100] = np.float32(1e-36)
    for row in x:
        y, ref = ctx.matmul(gtype, wq, row[None], n, k)[0], w @ row.astype(np.float64)
        assert np.all(np.abs(y - ref) <= 1e-6 * np.abs(ref).max() + 3e-45)


# One infinity, or one that is no number, used to have every result formed again, value by value, by one thread each: 14 to 41 times as long.
@pytest.mark.parametrize("tname", sorted(TYPES))
@pytest.mark.parametrize("m", [1, 2])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_rows_that_are_not_finite_take_no_other_way(ctx, tname, m, bad):
    gtype, otype = TYPES[tname]
    n, k = 8192, 4096
    wb = ctx.buf(normal_weights(1, n, k, otype), mx.DType.U8)
    yb = ctx.device.alloc_buffer(m * n * 4, mx.DType.F32)
    x = normal_acts(m, m, k)
    times = []
    for row in (x, np.where(np.arange(k) == 77, np.float32(bad), x)):
        xb = ctx.buf(row.astype(np.float32), mx.DType.F32)
        took = []
        for _ in range(8):
            enc = ctx.device.command_encoder()
            mx.quantized_matmul_ggml(enc, ctx.registry, ctx.device, xb, wb, yb, mx.GgmlQuantizedMatmulParams(m, n, k, gtype))
            took.append(enc.commit_wait_with_gpu_time())
        times.append(min(took))
    assert mx.last_kernel_name() == "qmv_split"
    assert not np.isfinite(yb.as_slice(np.float32)).any()
    assert times[1] <= 5 * times[0]


@pytest.mark.parametrize("tname,n,k,m", [("Q4_0", 28500, 256, 3), ("Q8_0", 28449, 96, 4), ("Q4_0", 28300, 256, 4)])
def test_three_and_four_rows_of_many_tiles(ctx, tname, n, k, m):
    """Many chunks for every cluster, dealt out in turn; a last one that is part-filled."""
    gtype, otype = ALL[tname]
    wq = normal_weights(n + k, n, k, otype)
    x = normal_acts(n + m, m, k)
    y = ctx.matmul(gtype, wq, x, n, k)
    assert mx.last_kernel_name() == "qmv_split"
    y_ref, ad = orc.qmatmul(otype, wq, x, n, k, nthreads=8)
    assert norm_err(y, y_ref, ad) <= MV_TOL
