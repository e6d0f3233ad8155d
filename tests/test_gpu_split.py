"""The split mat-vec (csrc/qmv_split.cuh) at the edges of its tiles, slices, alignments and row groups, against the oracle."""
import numpy as np
import pytest

import mlx_native_b200 as mx
from oracle import oracle as orc
from tests.gpu_util import MV_TOL, TYPES, Ctx, norm_err, normal_acts, normal_weights
from tests.test_oracle_q5k import random_q5k_blocks

pytestmark = pytest.mark.gpu
ALL = dict(TYPES, Q4_K=(mx.GgmlType.Q4_K, orc.Q4_K))


@pytest.fixture(scope="module")
def ctx():
    mx.set_option("qmv", "split")          # wherever it can, not only where it is the faster kernel
    yield Ctx()
    mx.set_option("qmv", "auto")


# 16-row tiles, units of 64 values, slices of 256 over up to 8 ranks, sets of 4 activation rows; K that is no multiple of 256
# (rows at any even address), of 64 (half a unit), or shorter than a slice
@pytest.mark.parametrize("tname,n,k,m", [
    ("Q4_0", 1, 32, 1), ("Q4_0", 17, 96, 2), ("Q4_0", 15, 256, 3), ("Q4_0", 333, 2880, 5), ("Q4_0", 64, 4096, 8), ("Q4_0", 2500, 1056, 1),
    ("Q4_0", 12000, 4128, 8),                                      # several chunks per cluster: every receive buffer used again
    ("Q8_0", 1, 32, 8), ("Q8_0", 31, 160, 1), ("Q8_0", 2873, 2880, 5), ("Q8_0", 48, 512, 4), ("Q8_0", 130, 12288, 8), ("Q8_0", 1030, 4128, 2),
    ("Q6_K", 1, 256, 1), ("Q6_K", 33, 768, 7), ("Q6_K", 70, 2048, 2), ("Q6_K", 19, 5120, 8), ("Q6_K", 1001, 2560, 1), ("Q6_K", 12, 14336, 3),
    ("Q4_K", 16, 256, 1), ("Q4_K", 65, 768, 6), ("Q4_K", 40, 3584, 4), ("Q4_K", 130, 1024, 9), ("Q4_K", 50, 2304, 33),
    # eight columns where four slices of K do not fit and eight leave the last rank without work
    ("Q4_0", 40, 10304, 5), ("Q4_0", 21, 12544, 8), ("Q8_0", 33, 12352, 8), ("Q8_0", 18, 10752, 5), ("Q6_K", 20, 12544, 8), ("Q6_K", 37, 10496, 5),
    ("Q4_K", 24, 10752, 8), ("Q4_K", 24, 10496, 40), ("Q4_K", 17, 12544, 5)])
def test_dense(ctx, tname, n, k, m):
    gtype, otype = ALL[tname]
    wq = normal_weights(n + k + m, n, k, otype)
    x = normal_acts(n + m, m, k)
    x[:, ::7] *= 1e-4          # (one power-of-two scale per row and slice)
    y = ctx.matmul(gtype, wq, x, n, k)
    assert mx.last_kernel_name() == "qmv_split"
    y_ref, ad = orc.qmatmul(otype, wq, x, n, k, nthreads=8)
    assert norm_err(y, y_ref, ad) <= MV_TOL
    assert np.array_equal(y.view(np.uint32), ctx.matmul(gtype, wq, x, n, k).view(np.uint32))


@pytest.mark.parametrize("tname,offset", [("Q4_0", 2), ("Q4_0", 12), ("Q8_0", 6), ("Q8_0", 14), ("Q6_K", 2), ("Q6_K", 10)])
@pytest.mark.parametrize("m", [1, 6])
def test_weights_at_any_even_address(ctx, tname, offset, m):
    gtype, otype = TYPES[tname]
    n, k = 77, 2048
    wq = normal_weights(5, n, k, otype)
    big = np.zeros(wq.size + 64, np.uint8)
    big[offset:offset + wq.size] = wq
    x = normal_acts(1, m, k)
    y = ctx.matmul(gtype, wq, x, n, k, weight_buf=ctx.buf(big, mx.DType.U8).slice_view(offset, wq.size))
    assert mx.last_kernel_name() == "qmv_split"
    y_ref, ad = orc.qmatmul(otype, wq, x, n, k)
    assert norm_err(y, y_ref, ad) <= MV_TOL


# routed: experts without rows, with one row, with more than a pass takes (4); ids that name no expert; aligned rows and not
@pytest.mark.parametrize("tname,T,top_k,E,n,k", [
    ("Q4_0", 1, 8, 16, 40, 512), ("Q4_0", 32, 8, 8, 65, 288), ("Q8_0", 24, 8, 128, 48, 768), ("Q8_0", 7, 3, 5, 17, 96), ("Q6_K", 20, 4, 6, 50, 768),
    ("Q6_K", 3, 1, 4, 130, 2048), ("Q4_K", 32, 4, 16, 33, 2048), ("Q5_K", 9, 8, 32, 100, 512), ("Q5_K", 32, 8, 4, 16, 256)])
def test_routed(ctx, tname, T, top_k, E, n, k):
    rng = np.random.default_rng(T * 100 + n)
    if tname == "Q5_K":
        gtype, otype = mx.GgmlType.Q5_K, orc.Q5_K
        w = random_q5k_blocks(rng, E * n * (k // 256))
    else:
        gtype, otype = ALL[tname]
        w = normal_weights(E + n, E * n, k, otype)
    x = normal_acts(T, T, k)
    ids = rng.integers(0, E, T * top_k).astype(np.uint32)
    bad = np.zeros(ids.size, bool)
    if ids.size > 20:
        bad[[5, 11]] = True
    y, _ = ctx.matmul_id(gtype, w, w.size // E, x, np.where(bad, 0xFFFFFFFF, ids).astype(np.uint32), top_k, n, k, E)
    assert mx.last_kernel_name() == "qmv_split"
    y_ref, ad = orc.qmatmul_id(otype, w, w.size // E, x, ids, top_k, n, k, E, nthreads=8)
    assert norm_err(y[~bad], y_ref[~bad], ad[~bad]) <= MV_TOL
    assert np.all(y[bad] == 0)


# a single pair: passes of activations that stay in registers and those loaded again, aligned rows and not, infinities and large numbers
@pytest.mark.parametrize("tname,n,k", [("Q4_0", 40, 96), ("Q4_0", 33, 2080), ("Q4_0", 48, 8192), ("Q8_0", 20, 16640), ("Q8_0", 34, 1088), ("Q6_K", 18, 2560), ("Q6_K", 33, 16384),
                                       ("Q4_K", 50, 4352), ("Q5_K", 24, 2304)])
def test_routed_single_pair(ctx, tname, n, k):
    E = 3
    if tname == "Q5_K":
        gtype, otype = mx.GgmlType.Q5_K, orc.Q5_K
        w = random_q5k_blocks(np.random.default_rng(n), E * n * (k // 256))
    else:
        gtype, otype = ALL[tname]
        w = normal_weights(E + n, E * n, k, otype)
    for i, x in enumerate(extreme_rows(k, 1e30)):
        ids = np.array([i % E], np.uint32)
        y, _ = ctx.matmul_id(gtype, w, w.size // E, x[None], ids, 1, n, k, E)
        assert mx.last_kernel_name() == "qmv_split"
        y_ref, ad = orc.qmatmul_id(otype, w, w.size // E, x[None], ids, 1, n, k, E)
        assert_same_numbers(y, y_ref, ad)


def test_batch_of_different_shapes(ctx):
    """Mat-vecs of one launch that differ in rows, K (ranks without work for the shorter one), activations and row count."""
    gtype, otype = TYPES["Q8_0"]
    d = ctx.device
    shapes = [(100, 4096, 8), (33, 512, 5), (16, 4096, 7), (257, 1024, 8)]
    ws = [normal_weights(i, n, k, otype) for i, (n, k, m) in enumerate(shapes)]
    xs = [normal_acts(i, m, k) for i, (n, k, m) in enumerate(shapes)]
    bufs = [(ctx.buf(x, mx.DType.F32), ctx.buf(w, mx.DType.U8), d.alloc_buffer(m * n * 4, mx.DType.F32)) for x, w, (n, k, m) in zip(xs, ws, shapes)]
    mx.reset_counters()
    enc = d.command_encoder()
    for (xb, wb, yb), (n, k, m) in zip(bufs, shapes):
        mx.quantized_matmul_ggml(enc, ctx.registry, d, xb, wb, yb, mx.GgmlQuantizedMatmulParams(m, n, k, gtype))
    enc.commit_and_wait()
    assert mx.last_kernel_name() == "qmv_split"
    assert mx.kernel_launch_count() == 2          # the activations of all of them packed by one kernel, then one mat-vec kernel
    for (xb, wb, yb), w, x, (n, k, m) in zip(bufs, ws, xs, shapes):
        y_ref, ad = orc.qmatmul(otype, w, x, n, k)
        assert norm_err(yb.as_slice(np.float32).reshape(m, n), y_ref, ad) <= MV_TOL


# Every product of a code and an f16 half is exact, a half pair holds 22 bits, and the f32 sums of a result have at most a few dozen
# terms one after another: relative 2-norm errors of 1 to 1.5e-7 (2^-23 = 1.2e-7), also where a few activations are 300 times larger than the
# others.  (Codes multiplied as subnormals miss this bound by 2 (Q8_0) to 20 times.)
ERR_TOL = 5e-7


def relative_error(y, w, x):
    ref = x.astype(np.float64) @ w.T
    return np.linalg.norm(y - ref) / np.linalg.norm(ref)


@pytest.mark.parametrize("rows", [1, 4, 8])
@pytest.mark.parametrize("tname,n,k", [("Q4_0", 700, 2880), ("Q4_0", 700, 4096), ("Q8_0", 700, 2880), ("Q8_0", 700, 4096), ("Q6_K", 700, 2816),
                                       ("Q6_K", 700, 4096), ("Q4_K", 700, 4096)])
def test_error_against_64_bits(ctx, tname, n, k, rows):
    gtype, otype = ALL[tname]
    wq = normal_weights(n + k, n, k, otype)
    x = normal_acts(n + rows, rows, k)
    x[:, ::97] *= 300
    y = ctx.matmul(gtype, wq, x, n, k)
    assert mx.last_kernel_name() == "qmv_split"
    assert relative_error(y, orc.dequantize(otype, wq).reshape(n, k).astype(np.float64), x) <= ERR_TOL


# activation rows that f16 halves could lose: infinities, no numbers, magnitudes at either end of f32
def extreme_rows(k, top=1e36):
    x = normal_acts(k, 7, k)
    x[0, 5] = np.inf
    x[1, k - 3] = -np.inf
    x[2, [1, 9, k - 20]] = [np.inf, -np.inf, 3.0]
    x[3, 17] = np.nan
    x[4] *= top
    x[5] *= 1e-35
    x[6, 30] = 4e4
    return x


def assert_same_numbers(y, y_ref, ad):
    assert np.array_equal(np.isnan(y), np.isnan(y_ref))
    inf = np.isinf(y_ref)
    assert np.array_equal(y[inf], y_ref[inf])
    ok = np.isfinite(y_ref)
    assert np.all(np.abs(y[ok].astype(np.float64) - y_ref[ok]) <= MV_TOL * ad[ok])


@pytest.mark.parametrize("rows", [1, 2, 7])
@pytest.mark.parametrize("tname,n,k", [("Q4_0", 33, 288), ("Q4_0", 40, 2048), ("Q8_0", 33, 288), ("Q8_0", 40, 2048), ("Q6_K", 33, 768),
                                       ("Q6_K", 40, 2048), ("Q4_K", 33, 768), ("Q4_K", 600, 4096)])
def test_infinities_and_extreme_magnitudes(ctx, tname, n, k, rows):
    gtype, otype = ALL[tname]
    wq = normal_weights(n + k, n, k, otype)
    x = extreme_rows(k)
    y_ref, ad = orc.qmatmul(otype, wq, x, n, k, nthreads=8)
    for at in range(0, 7, rows):
        assert_same_numbers(ctx.matmul(gtype, wq, x[at:at + rows], n, k), y_ref[at:at + rows], ad[at:at + rows])


@pytest.mark.parametrize("tname,n,k", [("Q4_0", 33, 288), ("Q8_0", 40, 2048), ("Q6_K", 33, 768), ("Q4_K", 33, 768), ("Q5_K", 18, 512)])
def test_routed_infinities_and_extreme_magnitudes(ctx, tname, n, k):
    T, top_k, E = 21, 2, 4
    rng = np.random.default_rng(n)
    if tname == "Q5_K":
        gtype, otype = mx.GgmlType.Q5_K, orc.Q5_K
        w = random_q5k_blocks(rng, E * n * (k // 256))
    else:
        gtype, otype = ALL[tname]
        w = normal_weights(E + n, E * n, k, otype)
    x = np.concatenate([extreme_rows(k, 1e30 if tname == "Q5_K" else 1e36)] * 3)   # (random Q5_K blocks hold large weights)
    ids = np.stack([rng.permutation(E)[:top_k] for _ in range(T)]).astype(np.uint32).reshape(-1)
    y, _ = ctx.matmul_id(gtype, w, w.size // E, x, ids, top_k, n, k, E)
    y_ref, ad = orc.qmatmul_id(otype, w, w.size // E, x, ids, top_k, n, k, E, nthreads=8)
    assert mx.last_kernel_name() == "qmv_split"
    assert_same_numbers(y, y_ref, ad)
