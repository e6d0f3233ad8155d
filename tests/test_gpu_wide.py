"""The Q4_K kernel for many activation rows (csrc/qmv_wide.cu) at the edges of its tiles (128 / 256 weight rows, 16 / 32 / 48 activation
rows) and of its K parts, against the oracle."""
import numpy as np
import pytest

import mlx_native_b200 as mx
from oracle import oracle as orc
from tests.gpu_util import MV_TOL, Ctx, norm_err, normal_acts, normal_weights
from tests.test_gpu_split import ERR_TOL, assert_same_numbers, extreme_rows, relative_error

pytestmark = pytest.mark.gpu
G, O = mx.GgmlType.Q4_K, orc.Q4_K


@pytest.fixture(scope="module")
def ctx():
    return Ctx()


# one tile and a bit of the next, one row short of a tile, K of one super-block, of an odd number, of fewer than the parts it could have;
# result rows that do not start on 16-byte boundaries
@pytest.mark.parametrize("n,k,m", [(4096, 256, 9), (4097, 256, 16), (1367, 768, 17), (512, 2048, 32), (129, 8192, 33), (385, 3328, 48), (4099, 256, 49),
                                   (255, 4352, 97), (2050, 1024, 200), (333, 14336, 11), (1500, 768, 513)])
def test_dense(ctx, n, k, m):
    wq = normal_weights(n + k + m, n, k, O)
    x = normal_acts(n + m, m, k)
    x[:, ::7] *= 1e-4
    y = ctx.matmul(G, wq, x, n, k)
    assert mx.last_kernel_name() == "qmv_wide"
    y_ref, ad = orc.qmatmul(O, wq, x, n, k, nthreads=8)
    assert norm_err(y, y_ref, ad) <= MV_TOL
    assert np.array_equal(y.view(np.uint32), ctx.matmul(G, wq, x, n, k).view(np.uint32))


@pytest.mark.parametrize("n,k,m", [(700, 4096, 40), (300, 14336, 70), (2100, 1024, 9)])
def test_error_against_64_bits(ctx, n, k, m):
    wq = normal_weights(n + k, n, k, O)
    x = normal_acts(n + m, m, k)
    x[:, ::97] *= 300
    y = ctx.matmul(G, wq, x, n, k)
    assert mx.last_kernel_name() == "qmv_wide"
    assert relative_error(y, orc.dequantize(O, wq).reshape(n, k).astype(np.float64), x) <= ERR_TOL


def test_infinities_and_extreme_magnitudes(ctx):
    n, k = 600, 2048
    wq = normal_weights(n + k, n, k, O)
    x = np.concatenate([extreme_rows(k), normal_acts(1, 20, k), extreme_rows(k)])
    y_ref, ad = orc.qmatmul(O, wq, x, n, k, nthreads=8)
    y = ctx.matmul(G, wq, x, n, k)
    assert mx.last_kernel_name() == "qmv_wide"
    assert_same_numbers(y, y_ref, ad)


def test_products_of_one_group_share_a_launch(ctx):
    """Three products of the same activations and one of others (other K too), between two barriers: one packing and one product kernel."""
    d, m = ctx.device, 21
    shapes = [(1100, 1024), (2048, 1024), (1025, 1024), (520, 2304)]
    ws = [normal_weights(i, n, k, O) for i, (n, k) in enumerate(shapes)]
    xs = {k: normal_acts(k, m, k) for k in (1024, 2304)}
    xb = {k: ctx.buf(x, mx.DType.F32) for k, x in xs.items()}
    bufs = [(ctx.buf(w, mx.DType.U8), d.alloc_buffer(m * n * 4, mx.DType.F32)) for w, (n, k) in zip(ws, shapes)]
    mx.reset_counters()
    enc = d.command_encoder()
    for (wb, yb), (n, k) in zip(bufs, shapes):
        mx.quantized_matmul_ggml(enc, ctx.registry, d, xb[k], wb, yb, mx.GgmlQuantizedMatmulParams(m, n, k, G))
    enc.commit_and_wait()
    assert mx.last_kernel_name() == "qmv_wide" and mx.kernel_launch_count() == 2
    for (wb, yb), w, (n, k) in zip(bufs, ws, shapes):
        y_ref, ad = orc.qmatmul(O, w, xs[k], n, k, nthreads=4)
        assert norm_err(yb.as_slice(np.float32).reshape(m, n), y_ref, ad) <= MV_TOL


def test_a_captured_group(ctx):
    """Recorded once, replayed on other activations and results of before."""
    d, m, n, k = ctx.device, 19, 1100, 1024
    ws = [normal_weights(i, n, k, O) for i in range(2)]
    xb = ctx.buf(normal_acts(1, m, k), mx.DType.F32)
    bufs = [(ctx.buf(w, mx.DType.U8), ctx.buf(np.zeros((m, n), np.float32), mx.DType.F32)) for w in ws]
    enc = d.command_encoder()

    def encode():
        for wb, yb in bufs:
            mx.quantized_matmul_ggml(enc, ctx.registry, d, xb, wb, yb, mx.GgmlQuantizedMatmulParams(m, n, k, G))

    encode()
    enc.commit_and_wait()
    enc.begin_capture()
    encode()
    graph = enc.end_capture()
    assert mx.last_kernel_name() == "qmv_wide"
    for seed in (2, 3):
        x = normal_acts(seed, m, k)
        xb.upload(x)
        graph.launch(enc)
        enc.commit_and_wait()
        for (_, yb), w in zip(bufs, ws):
            y_ref, ad = orc.qmatmul(O, w, x, n, k, nthreads=4)
            assert norm_err(yb.as_slice(np.float32).reshape(m, n), y_ref, ad) <= MV_TOL


def test_weights_off_16_byte_boundaries_take_another_kernel(ctx):
    n, k, m = 512, 2048, 12
    wq = normal_weights(9, n, k, O)
    big = np.zeros(wq.size + 32, np.uint8)
    big[4:4 + wq.size] = wq
    x = normal_acts(3, m, k)
    y = ctx.matmul(G, wq, x, n, k, weight_buf=ctx.buf(big, mx.DType.U8).slice_view(4, wq.size))
    assert mx.last_kernel_name() != "qmv_wide"
    y_ref, ad = orc.qmatmul(O, wq, x, n, k, nthreads=4)
    assert norm_err(y, y_ref, ad) <= MV_TOL
