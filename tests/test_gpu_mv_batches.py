"""Which kernel a batch of independent mat-vecs leaves by is decided when the batch is complete, for all of it."""
import itertools

import numpy as np
import pytest

import mlx_native_b200 as mx
from oracle import oracle as orc
from tests.gpu_util import MV_TOL, TYPES, Ctx, norm_err, normal_acts, normal_weights

pytestmark = pytest.mark.gpu
K = 4096


@pytest.fixture(scope="module")
def ctx():
    return Ctx()


def encode(ctx, gtype, ops):
    """ops: (weights, activations, rows of the matrix); results and kernel launches of one group."""
    d = ctx.device
    bufs = [(ctx.buf(x, mx.DType.F32), w, d.alloc_buffer(x.shape[0] * n * 4, mx.DType.F32)) for w, x, n in ops]
    enc = d.command_encoder()
    mx.reset_counters()
    for (xb, wb, yb), (_, x, n) in zip(bufs, ops):
        mx.quantized_matmul_ggml(enc, ctx.registry, d, xb, wb, yb, mx.GgmlQuantizedMatmulParams(x.shape[0], n, K, gtype))
    enc.commit_and_wait()
    return [yb.as_slice(np.float32).reshape(x.shape[0], n).copy() for (_, _, yb), (_, x, n) in zip(bufs, ops)], mx.kernel_launch_count()


# alone, the largest of these leaves by the split kernel and the others do not; together they are one launch, in any order
@pytest.mark.parametrize("tname,m", [("Q4_0", 1), ("Q8_0", 1), ("Q8_0", 2), ("Q6_K", 1), ("Q4_0", 4)])
def test_any_order_is_one_launch(ctx, tname, m):
    gtype, otype = TYPES[tname]
    part = normal_weights(m, 1024, K, otype)
    x = normal_acts(m, m, K)
    y_ref, ad = orc.qmatmul(otype, part, x, 1024, K, nthreads=8)
    whole = ctx.buf(np.tile(part, 12), mx.DType.U8)
    sizes = {n: whole.slice_view(0, part.size * (n // 1024)) for n in (1024, 4096, 12288)}
    for order in itertools.permutations(sizes):
        ys, launches = encode(ctx, gtype, [(sizes[n], x, n) for n in order])
        assert launches == 1, order
        for y, n in zip(ys, order):
            for at in range(0, n, 1024):
                assert norm_err(y[:, at:at + 1024], y_ref, ad) <= MV_TOL


# Q4_K, five to eight rows: the split kernel (a packing launch ahead), or the register-level kernel where the matrix fills its passes.  More rows: the
# kernel for many rows, packing and product, whatever the matrix fills.
@pytest.mark.parametrize("m,n,launches,kernel", [(5, 1024, 2, "qmv_split"), (8, 16384, 1, "qmv_mma"), (16, 1024, 2, "qmv_wide"), (9, 1024, 2, "qmv_wide"),
                                                 (9, 8192, 2, "qmv_wide"), (24, 16384, 2, "qmv_wide")])
def test_q4k_of_many_rows(ctx, m, n, launches, kernel):
    part = normal_weights(n, 1024, K, orc.Q4_K)
    x = normal_acts(m, m, K)
    y_ref, ad = orc.qmatmul(orc.Q4_K, part, x, 1024, K, nthreads=8)
    (y,), count = encode(ctx, mx.GgmlType.Q4_K, [(ctx.buf(np.tile(part, n // 1024), mx.DType.U8), x, n)])
    assert count == launches and mx.last_kernel_name() == kernel
    for at in range(0, n, 1024):
        assert norm_err(y[:, at:at + 1024], y_ref, ad) <= MV_TOL


# a pair's sum does not depend on how many pairs the launch has, on either side of the number that one launch of the other kernel takes
@pytest.mark.parametrize("tname,n,k", [("Q4_0", 768, 2048), ("Q6_K", 768, 2048), ("Q8_0", 1024, 768), ("Q4_0", 512, 1024)])
def test_routed_rows_of_few_pairs_have_the_same_bits(ctx, tname, n, k):
    gtype, otype = TYPES[tname]
    E = 8
    w = normal_weights(n, E * n, k, otype)
    x = normal_acts(k, 16, k)
    ids = np.random.default_rng(n).integers(0, E, 16).astype(np.uint32)
    whole, _ = ctx.matmul_id(gtype, w, w.size // E, x, ids, 1, n, k, E)
    for rows in (1, 3, 8, 15):
        some, _ = ctx.matmul_id(gtype, w, w.size // E, x[:rows], ids[:rows], 1, n, k, E)
        assert np.array_equal(some.view(np.uint32), whole[:rows].view(np.uint32)), rows


# one and two rows: on either side of the lines between the register-level and the split kernel (csrc/qmv_split.cu: qmv_split_pays)
@pytest.mark.parametrize("tname,m,n,k,kernel", [
    ("Q8_0", 2, 20480, 4096, "qmv_split"), ("Q8_0", 2, 32768, 4096, "qmv_mma"), ("Q6_K", 2, 10240, 4096, "qmv_split"), ("Q6_K", 2, 18432, 4096, "qmv_mma"),
    ("Q6_K", 2, 14336, 4096, "qmv_split"), ("Q6_K", 2, 49152, 1024, "qmv_mma"), ("Q8_0", 1, 8192, 12288, "qmv_mma"), ("Q8_0", 1, 16384, 4096, "qmv_split"),
    ("Q8_0", 1, 10240, 4096, "qmv_split"), ("Q4_0", 2, 8192, 12288, "qmv_mma"), ("Q4_0", 2, 8192, 8192, "qmv_split")])
def test_where_one_and_two_rows_leave(ctx, tname, m, n, k, kernel):
    gtype, otype = TYPES[tname]
    part = normal_weights(n, 1024, k, otype)
    x = normal_acts(m, m, k)
    y_ref, ad = orc.qmatmul(otype, part, x, 1024, k, nthreads=8)
    y = ctx.matmul(gtype, np.tile(part, n // 1024), x, n, k)
    assert mx.last_kernel_name() == kernel
    for at in range(0, n, 1024):
        assert norm_err(y[:, at:at + 1024], y_ref, ad) <= MV_TOL
