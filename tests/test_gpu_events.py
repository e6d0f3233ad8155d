"""What a commit records: the end of a command buffer with and without its GPU time, in any order; lanes that fork after a batch of mat-vecs."""
import numpy as np
import pytest

import mlx_native_b200 as mx
from oracle import oracle as orc
from tests.gpu_util import MV_TOL, Ctx, norm_err, normal_acts, normal_weights

pytestmark = pytest.mark.gpu
G, O = mx.GgmlType.Q8_0, orc.Q8_0


@pytest.fixture(scope="module")
def ctx():
    return Ctx()


def test_gpu_time_beside_plain_commits(ctx):
    d, n, k = ctx.device, 256, 1024
    wq, x = normal_weights(1, n, k, O), normal_acts(1, 1, k)
    xb, wb, yb = ctx.buf(x, mx.DType.F32), ctx.buf(wq, mx.DType.U8), d.alloc_buffer(n * 4, mx.DType.F32)
    y_ref, ad = orc.qmatmul(O, wq, x, n, k)
    enc = d.command_encoder()
    for how in ("plain", "timed", "plain", "plain then timed", "split", "timed"):
        yb.as_mut_slice(np.float32)[:] = 0
        mx.quantized_matmul_ggml(enc, ctx.registry, d, xb, wb, yb, mx.GgmlQuantizedMatmulParams(1, n, k, G))
        if how == "plain":
            enc.commit_and_wait()
        elif how == "split":
            enc.commit()
            enc.wait_until_completed()
        else:
            if how == "plain then timed":
                enc.commit()
            assert 0 < enc.commit_wait_with_gpu_time() < 1
        assert norm_err(yb.as_slice(np.float32).reshape(1, n), y_ref, ad) <= MV_TOL, how


# The first operation of a group waits in the batch; the next runs at once on the other lane, one after that reads what an earlier group
# wrote.  Every kernel of a later group writes over what one of the group before reads.
@pytest.mark.parametrize("capture", [False, True])
def test_lanes_fork_behind_a_batch(ctx, capture):
    d, n = ctx.device, 2048
    wq = normal_weights(5, n, n, O)
    wb = ctx.buf(wq, mx.DType.U8)
    xs = [normal_acts(i, 1, n) for i in range(2)]
    gate, up = normal_acts(7, 1, n), normal_acts(8, 1, n)
    bufs = {k: ctx.buf(v, mx.DType.F32) for k, v in (("a", xs[0]), ("g", gate), ("u", up))}
    for k in ("b", "s", "t"):
        bufs[k] = d.alloc_buffer(n * 4, mx.DType.F32)
    p = mx.GgmlQuantizedMatmulParams(1, n, n, G)
    enc = d.command_encoder()

    def encode():
        for _ in range(5):
            mx.quantized_matmul_ggml(enc, ctx.registry, d, bufs["a"], wb, bufs["b"], p)   # waits in the batch
            mx.silu_mul(enc, ctx.registry, d, bufs["g"], bufs["u"], bufs["s"], n)         # other lane
            mx.silu_mul(enc, ctx.registry, d, bufs["s"], bufs["u"], bufs["t"], n)         # conflict: a new group
            mx.quantized_matmul_ggml(enc, ctx.registry, d, bufs["t"], wb, bufs["s"], p)   # reads t, writes over s

    if capture:
        for k in ("a", "g", "u"):   # uploaded before the recording
            mx.silu_mul(enc, ctx.registry, d, bufs[k], bufs[k], bufs["t"], n)
        enc.commit_and_wait()
        enc.begin_capture()
        encode()
        graph = enc.end_capture()
        graph.launch(enc)
    else:
        encode()
    enc.commit_and_wait()
    silu = lambda g, u: (g / (1 + np.exp(-g.astype(np.float64))) * u).astype(np.float32)
    t = silu(silu(gate, up), up)
    for name, x in (("b", xs[0]), ("s", t)):
        y_ref, ad = orc.qmatmul(O, wq, x, n, n, nthreads=4)
        # (silu's own rounding, 2^-22 of each value, besides the product's)
        assert norm_err(bufs[name].as_slice(np.float32).reshape(1, n), y_ref, ad) <= 2 * MV_TOL, name
